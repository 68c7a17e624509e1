// mlp.cu -- the learned warm start's multilayer perceptron on the tensor
// cores: a generic BF16 GEMM, the fused persistent inference kernel (the hot
// path: features -> 4 layers -> x0 update), the fused forward and backward
// pass of training, and Adam.
//
// The reference has no learned component; this is new functionality.  All
// matrix products run as tcgen05.mma (kind::f16, BF16 operands in shared
// memory, FP32 accumulators in tensor memory).
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <vector>

#include "engine.h"
#include "tc05.cuh"

using bf16 = __nv_bfloat16;

namespace avbd {
namespace {

constexpr unsigned HID = AVBD_MLP_HIDDEN;    // 128
constexpr unsigned IN = AVBD_MLP_IN_PAD;     // 32
constexpr unsigned OUT = AVBD_MLP_OUT_PAD;   // 16
// offsets of the flat parameter array
constexpr unsigned OFF_W1 = 0, OFF_B1 = 4096, OFF_W2 = 4224, OFF_B2 = 20608, OFF_W3 = 20736, OFF_B3 = 37120,
                   OFF_W4 = 37248, OFF_B4 = 39296, NPAR = AVBD_MLP_NPARAMS;
static_assert(OFF_B1 == HID * IN && OFF_W2 == OFF_B1 + HID && OFF_B2 == OFF_W2 + HID * HID &&
                  OFF_W3 == OFF_B2 + HID && OFF_B3 == OFF_W3 + HID * HID && OFF_W4 == OFF_B3 + HID &&
                  OFF_B4 == OFF_W4 + OUT * HID && NPAR == OFF_B4 + OUT,
              "parameter layout");

AVBD_D float silu(float z) { return z / (1.0f + __expf(-z)); }
// The same function as z/2 (1 + tanh(z/2)) with the hardware tanh
// approximation (one special-function operation instead of two; its error,
// about 2^-11 relative, is below the BF16 rounding of the result).
// h = z / 2.
AVBD_D float silu_half(float h) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h));
    return fmaf(h, t, h);
}
AVBD_D float silu_grad(float z) {
    float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}
AVBD_D uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

// R x K row-major BF16 global matrix (row stride ld) -> K-major canonical
// shared layout; rows >= rows_valid are zero
AVBD_D void load_kmaj(uint8_t* dst, const bf16* src, unsigned ld, unsigned R, unsigned K, unsigned rows_valid,
                      unsigned tid, unsigned nthreads) {
    const unsigned pieces = R * (K / 8);
    for (unsigned i = tid; i < pieces; i += nthreads) {
        const unsigned r = i % R, c = i / R;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < rows_valid) v = __ldg(reinterpret_cast<const uint4*>(src + (size_t)r * ld + c * 8));
        *reinterpret_cast<uint4*>(dst + c * (R * 16) + r * 16) = v;
    }
}

// Polls a barrier wait may take before it gives up (avbd_debug_set_wait_limit
// lowers it so that tests can make the wait run out).
__device__ uint32_t g_wait_polls = AVBD_DEFAULT_WAIT_POLLS;
// Polls the drain after a timeout may take: the MMAs already issued must
// land before the CTA frees the TMEM columns they write.
constexpr uint32_t kDrainPolls = AVBD_DEFAULT_WAIT_POLLS;

// all threads wait for the barrier phase; false (uniformly) if it timed out
AVBD_D bool block_wait(uint64_t* bar, uint32_t& phase) {
    bool got = tc::mbar_wait(bar, phase, *(volatile uint32_t*)&g_wait_polls);
    phase ^= 1u;
    return __syncthreads_and(got ? 1 : 0) != 0;
}

// After a wait gave up (phase already flipped by block_wait): wait, bounded,
// for the commit of the MMAs still in flight, so that no tensor-core write
// reaches the TMEM columns after they are freed.
AVBD_D void drain_after_timeout(uint64_t* bar, uint32_t phase) {
    if (threadIdx.x == 0) tc::mbar_wait(bar, phase ^ 1u, kDrainPolls);
    __syncthreads();
}

// one thread: D (+)= A B^T over `ksteps` K = 16 steps of two canonical operands
AVBD_D void issue(uint32_t d, uint32_t a, uint32_t a_rows, uint32_t b, uint32_t b_rows, unsigned ksteps,
                  uint32_t idesc, bool acc_first) {
    for (unsigned s = 0; s < ksteps; s++) {
        uint64_t da = tc::sdesc(a + s * 2 * a_rows * 16, a_rows * 16, 128);
        uint64_t db = tc::sdesc(b + s * 2 * b_rows * 16, b_rows * 16, 128);
        tc::mma_bf16(d, da, db, idesc, (acc_first || s > 0) ? 1u : 0u);
    }
}

// ------------------------------------------------------------ generic GEMM
// C [M x N] (+)= A [M x K] B [N x K]^T.  One CTA: 128 rows x NT columns, a
// K range of `kper` (split-K over blockIdx.z, atomics when split), K chunks
// of 64 staged in shared memory.
template <int NT>
__global__ void __launch_bounds__(128) k_gemm(const bf16* __restrict__ A, unsigned lda, const bf16* __restrict__ B,
                                              unsigned ldb, float* C, unsigned ldc, unsigned M, unsigned N, unsigned K,
                                              unsigned kper, int mode, int* err) {
    __shared__ __align__(1024) uint8_t sA[128 * 64 * 2];
    __shared__ __align__(1024) uint8_t sB[NT * 64 * 2];
    __shared__ uint64_t bar;
    __shared__ uint32_t tslot;
    constexpr uint32_t TCOLS = NT < 32 ? 32 : NT;
    const unsigned tid = threadIdx.x, warp = tid >> 5;
    const unsigned row0 = blockIdx.x * 128, col0 = blockIdx.y * NT;
    const unsigned kb = blockIdx.z * kper, ke = min(K, kb + kper);
    if (warp == 0) tc::tmem_alloc(&tslot, TCOLS);
    if (tid == 0) tc::mbar_init(&bar, 1);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tslot;
    const uint32_t idesc = tc::idesc_bf16(128, NT);
    const unsigned mrows = M > row0 ? min(128u, M - row0) : 0u;
    const unsigned nrows = N > col0 ? min((unsigned)NT, N - col0) : 0u;
    uint32_t phase = 0;
    bool ok = true;
    for (unsigned k0 = kb; k0 < ke && ok; k0 += 64) {
        const unsigned kl = min(64u, ke - k0);  // a multiple of 16
        load_kmaj(sA, A + (size_t)row0 * lda + k0, lda, 128, kl, mrows, tid, 128);
        load_kmaj(sB, B + (size_t)col0 * ldb + k0, ldb, NT, kl, nrows, tid, 128);
        tc::fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after();
            issue(tmem, tc::smem_u32(sA), 128, tc::smem_u32(sB), NT, kl / 16, idesc, k0 > kb);
            tc::commit(&bar);
        }
        ok = block_wait(&bar, phase);
    }
    if (!ok) drain_after_timeout(&bar, phase);
    tc::fence_after();
    if (ok && ke > kb) {
        const unsigned r = warp * 32 + (tid & 31);
        const unsigned gr = row0 + r;
#pragma unroll
        for (unsigned c = 0; c < (unsigned)NT; c += 16) {
            float v[16];
            tc::tmem_ld16(tmem + ((warp * 32u) << 16) + c, v);
            if (gr < M) {
                float* dst = C + (size_t)gr * ldc + col0 + c;
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    if (col0 + c + j >= N) break;
                    if (mode == 0) dst[j] = v[j];
                    else if (mode == 1) dst[j] += v[j];
                    else atomicAdd(dst + j, v[j]);
                }
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tmem_dealloc(tmem, TCOLS);
        tc::tmem_relinquish();
    }
    if (!ok && tid == 0) atomicExch(err, (int)AVBD_ERR_BARRIER_TIMEOUT);
}

}  // namespace

// C = A B^T (+ C): tile width from N, split-K when there are too few tiles
int gemm_bf16(const bf16* A, unsigned lda, const bf16* B, unsigned ldb, float* C, unsigned ldc, unsigned M,
              unsigned N, unsigned K, bool accumulate, cudaStream_t st, int* err) {
    if (M == 0 || N == 0 || K == 0) return AVBD_OK;
    if (K % 16 || lda % 8 || ldb % 8 || ((uintptr_t)A & 15) || ((uintptr_t)B & 15))
        return set_error(AVBD_ERR_INVALID_ARG, "gemm: K % 16, lda % 8, ldb % 8 and 16-byte aligned operands required");
    const unsigned NT = N <= 16 ? 16 : (N <= 32 ? 32 : 128);
    const unsigned mt = (M + 127) / 128, nt = (N + NT - 1) / NT;
    unsigned split = 1;
    if (mt * nt < 148 && K >= 512) split = std::min(K / 256, std::max(1u, 148u / (mt * nt)));
    unsigned kper = ((K + split - 1) / split + 63) / 64 * 64;
    split = (K + kper - 1) / kper;
    int mode = accumulate ? 1 : 0;
    if (split > 1) {  // partial sums are added atomically into a zeroed C
        if (!accumulate) {
            cudaError_t e = cudaMemset2DAsync(C, sizeof(float) * ldc, 0, sizeof(float) * N, M, st);
            if (e != cudaSuccess) return set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
        }
        mode = 2;
    }
    dim3 grid(mt, nt, split);
    if (NT == 16) k_gemm<16><<<grid, 128, 0, st>>>(A, lda, B, ldb, C, ldc, M, N, K, kper, mode, err);
    else if (NT == 32) k_gemm<32><<<grid, 128, 0, st>>>(A, lda, B, ldb, C, ldc, M, N, K, kper, mode, err);
    // 128-column tiles: 15 KB of unused dynamic shared memory caps residency at
    // 4 CTAs per SM, so their TMEM (4 x 128 columns) always fits at once
    else k_gemm<128><<<grid, 128, 15360, st>>>(A, lda, B, ldb, C, ldc, M, N, K, kper, mode, err);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AVBD_OK : set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
}

// ------------------------------------------------------ fused inference
namespace {

struct MlpW {
    const bf16 *w1, *w2, *w3, *w4;
    const float* b;  // b1 | b2 | b3 | b4 (400 floats)
};

// Where the outputs go: a plain FP32 array (out != null) or the solver
// state (x0 += scale * y for internal vertex `row`, with the iteration
// history x_last / x_lastlast reset to the new guess).
template <typename P>
struct MlpSink {
    float* out;
    typename Vec4Of<P>::T *x, *xl, *xll;
    const uint8_t* flags;  // row = internal vertex; fixed and oriented vertices are skipped
    P scale;
    float kappa;           // relative error assumed by the acceptance test
    unsigned long long* applied;  // count of accepted corrections (may be null)
};

// Thread groups of the fused inference: each takes its own tile through the
// layers with its own buffers (X: 2 x 8 KB, H: 32 KB), accumulator and
// barriers; the weights are shared.
constexpr unsigned GROUPS = 3, GTHREADS = 256;
constexpr unsigned SM_W1 = 0, SM_W2 = 8192, SM_W3 = 40960, SM_W4 = 73728, SM_X = 77824,
                   SM_H = SM_X + GROUPS * 16384, SM_BIAS = SM_H + GROUPS * 32768, SM_BAR = SM_BIAS + 1600,
                   SM_TSLOT = SM_BAR + 8 * GROUPS, SM_TOTAL = SM_TSLOT + 8;

// Feature tile (128 rows x 32 BF16) -> canonical K-major shared layout with
// cp.async (rows >= rows_valid are zero-filled), so the next tile streams in
// while this one runs through the layers.
AVBD_D void load_x_async(uint8_t* dst, const bf16* src, unsigned rows_valid, unsigned tid, unsigned nthreads) {
    for (unsigned i = tid; i < 128 * (IN / 8); i += nthreads) {
        const unsigned r = i % 128, c = i / 128;
        const bool in = r < rows_valid;
        const bf16* g = in ? src + (size_t)r * IN + c * 8 : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst + c * (128 * 16) + r * 16)),
                     "l"(g), "r"(in ? 16 : 0)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// TMEM accumulator -> bias + SiLU -> BF16 into the H operand.  8 warps: warp w
// reads lanes 32 (w % 4).. (rows) and the column half w / 4.  hbias: half the
// biases, so that the tanh's argument (v + b) / 2 is one multiply-add.
AVBD_D void epilogue_hidden(uint32_t tacc, const float* hbias, uint8_t* H, unsigned warp, unsigned lane) {
    const unsigned q = warp & 3u, hf = warp >> 2;
    const unsigned r = q * 32 + lane;
    const uint32_t base = tacc + ((q * 32u) << 16);
#pragma unroll
    for (unsigned c = hf * 64; c < hf * 64 + 64; c += 16) {
        float v[16];
        tc::tmem_ld16(base + c, v);
        uint32_t pk[8];
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 b = *reinterpret_cast<const float4*>(hbias + c + j);
            pk[j / 2] = pack2(silu_half(fmaf(0.5f, v[j], b.x)), silu_half(fmaf(0.5f, v[j + 1], b.y)));
            pk[j / 2 + 1] = pack2(silu_half(fmaf(0.5f, v[j + 2], b.z)), silu_half(fmaf(0.5f, v[j + 3], b.w)));
        }
        *reinterpret_cast<uint4*>(H + (c / 8) * (128 * 16) + r * 16) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(H + (c / 8 + 1) * (128 * 16) + r * 16) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
}

AVBD_D void group_sync(unsigned g) { asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(GTHREADS) : "memory"); }
// the group's threads wait for its barrier's phase; false (for all of them) if it timed out
AVBD_D bool group_wait(uint64_t* bar, uint32_t& phase, unsigned g) {
    const uint32_t got = tc::mbar_wait(bar, phase, *(volatile uint32_t*)&g_wait_polls) ? 1u : 0u;
    phase ^= 1u;
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(all)
        : "r"(got), "r"(g + 1), "r"(GTHREADS)
        : "memory");
    return all != 0;
}

// Acceptance of the correction y (in units of s = g h^2) of one vertex.  The
// block residual at the inertial guess is r0 = |features 12-14| (units of
// m g, L1).  Applying y with a relative error kappa leaves a residual of
// about kappa * sum_a (1 + H_aa h^2 / m) |y_a| (features 18-20 hold
// log(1 + H_aa h^2 / m)), so the correction is applied only where it removes
// more residual than its error adds, and never below 1e-4 m g (a vertex in
// free flight, where the inertial guess is exact up to rounding).
constexpr float WS_GATE = 1e-4f;
AVBD_D bool accept(const uint8_t* Xs, unsigned r, const float* y, float kappa) {
    const bf16* f = reinterpret_cast<const bf16*>(Xs + tc::kmaj_off(r, 12, 128));
    const bf16* h = reinterpret_cast<const bf16*>(Xs + tc::kmaj_off(r, 16, 128));  // features 16..23
    const float r0 = fabsf(__bfloat162float(f[0])) + fabsf(__bfloat162float(f[1])) + fabsf(__bfloat162float(f[2]));
    const float added = kappa * (__expf(__bfloat162float(h[2])) * fabsf(y[0]) +
                                 __expf(__bfloat162float(h[3])) * fabsf(y[1]) +
                                 __expf(__bfloat162float(h[4])) * fabsf(y[2]));
    return r0 > WS_GATE && r0 > added;
}

// Persistent: one CTA per SM, weights resident in shared memory, 128 feature
// rows per tile and thread group.  Bound by the hidden epilogues (a tanh per
// activation: 3,072 cycles of the special-function units a tile).  The layers
// of one tile are a chain (product, accumulator read, SiLU, operand store,
// fences); with one tile in flight per SM a million rows took 336 us, three
// times the tanh bound.  Three groups of 8 warps, each with a tile of its own
// and no barrier in common, fill one another's waits.
//
// OUT16: sink.out is 16-byte aligned, which the entry point does not ask of its
// callers (as a branch in here the other form cost the aligned one 1.5 %).
template <typename P, bool OUT16>
__global__ void __launch_bounds__(GROUPS * GTHREADS, 1) k_mlp_apply(MlpW w, const bf16* __restrict__ feat, unsigned n,
                                                                    MlpSink<P> sink, int* err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    constexpr unsigned NT = GROUPS * GTHREADS;
    uint8_t* W1s = sm + SM_W1;
    uint8_t* W2s = sm + SM_W2;
    uint8_t* W3s = sm + SM_W3;
    uint8_t* W4s = sm + SM_W4;
    const unsigned g = threadIdx.x / GTHREADS, tid = threadIdx.x % GTHREADS, warp = tid >> 5, lane = tid & 31;
    uint8_t* Xbuf = sm + SM_X + g * 16384;  // two 8 KB tiles
    uint8_t* Hs = sm + SM_H + g * 32768;
    float* bias = reinterpret_cast<float*>(sm + SM_BIAS);  // halved for the hidden layers
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SM_BAR) + g;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + SM_TSLOT);

    load_kmaj(W1s, w.w1, IN, HID, IN, HID, threadIdx.x, NT);
    load_kmaj(W2s, w.w2, HID, HID, HID, HID, threadIdx.x, NT);
    load_kmaj(W3s, w.w3, HID, HID, HID, HID, threadIdx.x, NT);
    load_kmaj(W4s, w.w4, HID, OUT, HID, OUT, threadIdx.x, NT);
    for (unsigned i = threadIdx.x; i < 3 * HID + OUT; i += NT) bias[i] = i < 3 * HID ? 0.5f * w.b[i] : w.b[i];
    if (threadIdx.x < 32) tc::tmem_alloc(tslot, 512);
    if (tid == 0) tc::mbar_init(bar, 1);
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t acc = *tslot + g * 128;
    const uint32_t id_h = tc::idesc_bf16(128, HID), id_o = tc::idesc_bf16(128, OUT);
    const uint32_t aH = tc::smem_u32(Hs);
    uint32_t phase = 0;
    bool ok = true;
    const unsigned ntiles = (n + 127) / 128, step = gridDim.x * GROUPS, first = blockIdx.x + gridDim.x * g;
    if (first < ntiles) load_x_async(Xbuf, feat + (size_t)first * 128 * IN, min(128u, n - first * 128), tid, GTHREADS);
    unsigned buf = 0;
    for (unsigned tile = first; tile < ntiles; tile += step, buf ^= 1u) {
        const unsigned row0 = tile * 128;
        uint8_t* Xs = Xbuf + buf * 8192;
        const uint32_t aX = tc::smem_u32(Xs);
        const unsigned next = tile + step;
        if (next < ntiles) {  // the other buffer was last read by the previous tile, finished
            load_x_async(Xbuf + (buf ^ 1u) * 8192, feat + (size_t)next * 128 * IN, min(128u, n - next * 128), tid,
                         GTHREADS);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        // one layer: D = A W^T into the group's accumulator
        auto layer = [&](uint32_t a, const uint8_t* W, unsigned rows, unsigned ksteps, uint32_t id) {
            tc::fence_before();  // the accumulator's readers are done
            tc::fence_async_smem();
            group_sync(g);
            if (tid == 0) {
                tc::fence_after();
                issue(acc, a, 128, tc::smem_u32(W), rows, ksteps, id, false);
                tc::commit(bar);
            }
            const bool got = group_wait(bar, phase, g);
            tc::fence_after();
            return got;
        };
        if (!(ok = layer(aX, W1s, HID, IN / 16, id_h))) break;
        epilogue_hidden(acc, bias, Hs, warp, lane);
        if (!(ok = layer(aH, W2s, HID, HID / 16, id_h))) break;
        epilogue_hidden(acc, bias + HID, Hs, warp, lane);
        if (!(ok = layer(aH, W3s, HID, HID / 16, id_h))) break;
        epilogue_hidden(acc, bias + 2 * HID, Hs, warp, lane);
        if (!(ok = layer(aH, W4s, OUT, HID / 16, id_o))) break;
        if (warp < 4) {
            float v[16];
            tc::tmem_ld16(acc + ((warp * 32u) << 16), v);
            const unsigned row = row0 + warp * 32 + lane;
            if (row < n) {
                const float* b4 = bias + 3 * HID;
                if (sink.out) {
                    float* o = sink.out + (size_t)row * OUT;
#pragma unroll
                    for (int j = 0; j < (int)OUT; j++) v[j] += b4[j];
                    if constexpr (OUT16) {
#pragma unroll
                        for (int j = 0; j < (int)OUT; j += 4)
                            *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                    } else {
#pragma unroll
                        for (int j = 0; j < (int)OUT; j++) o[j] = v[j];
                    }
                } else if (!(sink.flags[row] & (VF_FIXED | VF_ORIENTED))) {
                    const float y[3] = {v[0] + b4[0], v[1] + b4[1], v[2] + b4[2]};
                    if (accept(Xs, warp * 32 + lane, y, sink.kappa)) {
                        if (sink.applied) atomicAdd(sink.applied, 1ull);
                        typename Vec4Of<P>::T x4 = sink.x[row];
                        x4.x += sink.scale * (P)y[0];
                        x4.y += sink.scale * (P)y[1];
                        x4.z += sink.scale * (P)y[2];
                        sink.x[row] = x4;
                        sink.xl[row] = x4;
                        sink.xll[row] = x4;
                    }
                }
            }
        }
        group_sync(g);  // Xs is refilled by the next tile's prefetch
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");  // no copy may land after the exit
    if (!ok && tid == 0) tc::mbar_wait(bar, phase ^ 1u, kDrainPolls);  // as drain_after_timeout
    tc::fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc::tmem_dealloc(*tslot, 512);
        tc::tmem_relinquish();
    }
    if (!ok && tid == 0) atomicExch(err, (int)AVBD_ERR_BARRIER_TIMEOUT);
}

// ------------------------------------------------------ training kernels
// Shared memory of the fused training pass: weights, the feature tile, the
// three activations (each overwritten by its layer's gradient in the backward
// pass), dY, biases, bias gradients.
constexpr unsigned TR_X = SM_X, TR_H = TR_X + 8192, TR_DY = TR_H + 3 * 32768, TR_BIAS = TR_DY + 4096,
                   TR_DB = TR_BIAS + 1600, TR_LOSS = TR_DB + 1600, TR_BAR = TR_LOSS + 8, TR_TSLOT = TR_BAR + 8,
                   TR_TOTAL = TR_TSLOT + 8;

// descriptors of the same stored matrix (rows r, columns c; R rows) as a
// K-major operand (K along c) and as an MN-major one (K along r)
AVBD_D uint64_t desc_k(uint32_t a, uint32_t R, unsigned step) { return tc::sdesc(a + step * 2 * R * 16, R * 16, 128); }
AVBD_D uint64_t desc_mn(uint32_t a, uint32_t R, unsigned step) { return tc::sdesc(a + step * 256, 128, R * 16); }

// Sums over a warp's 32 rows of 16 columns: halves are exchanged and kept, so
// that lane l ends with column (l / 2) of the 16 (16 shuffles instead of 80).
AVBD_D float column_sum16(const float (&d)[16], unsigned lane) {
    float a[8], b[4], e[2];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float keep = lane & 16u ? d[j + 8] : d[j], give = lane & 16u ? d[j] : d[j + 8];
        a[j] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float keep = lane & 8u ? a[j + 4] : a[j], give = lane & 8u ? a[j] : a[j + 4];
        b[j] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const float keep = lane & 4u ? b[j + 2] : b[j], give = lane & 4u ? b[j] : b[j + 2];
        e[j] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    }
    const float keep = lane & 2u ? e[1] : e[0], give = lane & 2u ? e[0] : e[1];
    const float f = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    return f + __shfl_xor_sync(0xffffffffu, f, 1);
}

AVBD_D void red_add4(float* p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

// Forward and backward of a mini-batch, 128 rows a tile, one CTA per SM: the
// pre-activations stay in tensor memory (3 x 128 FP32 columns, the fourth
// 128 take the output and the activation gradients), the activations in
// shared memory, and each weight gradient of the tile accumulates where its
// layer's pre-activations were, to be added to G with 16-byte reductions.
// The transposed operands (dZ^T, H^T, W) are the stored ones read MN-major.
// Replaces 26 launches that passed every layer through memory twice (once
// transposed), one of them with an atomic per element on 128 addresses: a
// mini-batch of 8,192 took 0.42 ms of them.
// loss = mean over rows and the 3 outputs of w (y - t)^2, w the row's weight
// (target column 3); precisions as in the separate kernels: Z, dH and the
// accumulators FP32, H, dY and dZ rounded to BF16, bias gradients summed from
// the unrounded FP32 values.
__global__ void __launch_bounds__(512, 1) k_train(MlpW w, const bf16* __restrict__ feat, const float* __restrict__ T,
                                                   unsigned B, float* __restrict__ G, float* loss, int* err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t *W1s = sm + SM_W1, *W2s = sm + SM_W2, *W3s = sm + SM_W3, *W4s = sm + SM_W4;
    uint8_t *Xs = sm + TR_X, *dYs = sm + TR_DY;
    uint8_t* Hs[3] = {sm + TR_H, sm + TR_H + 32768, sm + TR_H + 65536};
    float* bias = reinterpret_cast<float*>(sm + TR_BIAS);
    float* db = reinterpret_cast<float*>(sm + TR_DB);
    float* lsum = reinterpret_cast<float*>(sm + TR_LOSS);
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + TR_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + TR_TSLOT);
    const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    load_kmaj(W1s, w.w1, IN, HID, IN, HID, tid, 512);
    load_kmaj(W2s, w.w2, HID, HID, HID, HID, tid, 512);
    load_kmaj(W3s, w.w3, HID, HID, HID, HID, tid, 512);
    load_kmaj(W4s, w.w4, HID, OUT, HID, OUT, tid, 512);
    for (unsigned i = tid; i < 3 * HID + OUT; i += 512) {
        bias[i] = w.b[i];
        db[i] = 0.f;
    }
    if (tid == 0) *lsum = 0.f;
    if (warp == 0) tc::tmem_alloc(tslot, 512);
    if (tid == 0) tc::mbar_init(bar, 1);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot, work = tmem + 384;
    const uint32_t id_h = tc::idesc_bf16(128, HID), id_o = tc::idesc_bf16(128, OUT);
    const uint32_t id_hb = tc::idesc_bf16(128, HID, false, true);  // dH = dZ W: B MN-major
    const uint32_t id_w = tc::idesc_bf16(128, HID, true, true), id_w1 = tc::idesc_bf16(128, IN, true, true),
                   id_w4 = tc::idesc_bf16(128, OUT, true, true);   // dW: both MN-major
    // this thread's part of a 128 x 128 accumulator: row r, columns c0 .. c0 + 31
    const unsigned q = warp & 3u, c0 = (warp >> 2) * 32, r = q * 32 + lane;
    const uint32_t trow = (q * 32u) << 16;
    uint32_t phase = 0;
    bool ok = true;
    // operands written by all threads are ready and the accumulators read: issue, then wait
    auto run = [&](auto&& products, auto&& meanwhile) {
        tc::fence_before();
        tc::fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after();
            products();
            tc::commit(bar);
        }
        __syncwarp();
        meanwhile();
        ok = block_wait(bar, phase);
        tc::fence_after();
        return ok;
    };
    auto nothing = [] {};
    auto product = [&](uint32_t d, const uint8_t* A, bool a_mn, const uint8_t* Bm, unsigned b_rows, bool b_mn,
                       unsigned ksteps, uint32_t id) {
        const uint32_t a = tc::smem_u32(A), bb = tc::smem_u32(Bm);
        for (unsigned s = 0; s < ksteps; s++)
            tc::mma_bf16(d, a_mn ? desc_mn(a, 128, s) : desc_k(a, 128, s),
                         b_mn ? desc_mn(bb, b_rows, s) : desc_k(bb, b_rows, s), id, s > 0 ? 1u : 0u);
    };
    // hidden layer's activation: Z + b -> SiLU -> BF16 into H
    auto activate = [&](uint32_t z, const float* b, uint8_t* H) {
#pragma unroll
        for (unsigned c = 0; c < 32; c += 16) {
            float v[16];
            tc::tmem_ld16(z + trow + c0 + c, v);
            uint32_t pk[8];
#pragma unroll
            for (int j = 0; j < 8; j++)
                pk[j] = pack2(silu(v[2 * j] + b[c0 + c + 2 * j]), silu(v[2 * j + 1] + b[c0 + c + 2 * j + 1]));
            uint8_t* d = H + ((c0 + c) / 8) * 2048 + r * 16;
            *reinterpret_cast<uint4*>(d) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            *reinterpret_cast<uint4*>(d + 2048) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
    };
    // dZ = dH silu'(Z + b) -> BF16 into H's buffer; bias gradient
    auto activate_grad = [&](uint32_t z, const float* b, uint8_t* H, float* dbl) {
#pragma unroll
        for (unsigned c = 0; c < 32; c += 16) {
            float v[16], d[16];
            tc::tmem_ld16(z + trow + c0 + c, v);
            tc::tmem_ld16(work + trow + c0 + c, d);
#pragma unroll
            for (int j = 0; j < 16; j++) d[j] *= silu_grad(v[j] + b[c0 + c + j]);
            uint8_t* o = H + ((c0 + c) / 8) * 2048 + r * 16;
            *reinterpret_cast<uint4*>(o) = make_uint4(pack2(d[0], d[1]), pack2(d[2], d[3]), pack2(d[4], d[5]), pack2(d[6], d[7]));
            *reinterpret_cast<uint4*>(o + 2048) =
                make_uint4(pack2(d[8], d[9]), pack2(d[10], d[11]), pack2(d[12], d[13]), pack2(d[14], d[15]));
            const float t = column_sum16(d, lane);
            if (!(lane & 1u)) atomicAdd(dbl + c0 + c + (lane >> 1), t);
        }
    };
    // a tile's weight gradient [128][128] added to G
    auto flush = [&](uint32_t acc, float* g) {
#pragma unroll
        for (unsigned c = 0; c < 32; c += 16) {
            float v[16];
            tc::tmem_ld16(acc + trow + c0 + c, v);
#pragma unroll
            for (int j = 0; j < 16; j += 4) red_add4(g + r * HID + c0 + c + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
    };

    for (unsigned tile = blockIdx.x; tile < B / 128; tile += gridDim.x) {
        const unsigned row0 = tile * 128;
        load_x_async(Xs, feat + (size_t)row0 * IN, 128, tid, 512);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        // forward
        if (!run([&] { product(tmem, Xs, false, W1s, HID, false, IN / 16, id_h); }, nothing)) break;
        activate(tmem, bias, Hs[0]);
        if (!run([&] { product(tmem + 128, Hs[0], false, W2s, HID, false, HID / 16, id_h); }, nothing)) break;
        activate(tmem + 128, bias + HID, Hs[1]);
        if (!run([&] { product(tmem + 256, Hs[1], false, W3s, HID, false, HID / 16, id_h); }, nothing)) break;
        activate(tmem + 256, bias + 2 * HID, Hs[2]);
        if (!run([&] { product(work, Hs[2], false, W4s, OUT, false, HID / 16, id_o); }, nothing)) break;
        // loss, dY
        if (warp < 4) {
            float v[16], d[16];
            tc::tmem_ld16(work + trow, v);
            const float* t = T + (size_t)(row0 + r) * 4;
            const float wt = t[3];
            float l = 0.f;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                d[j] = 0.f;
                if (j < AVBD_MLP_OUT) {
                    const float e = (v[j] + bias[3 * HID + j]) - t[j];
                    l += wt * e * e;
                    d[j] = 2.0f * wt * e / (float)(B * AVBD_MLP_OUT);
                }
            }
            *reinterpret_cast<uint4*>(dYs + r * 16) =
                make_uint4(pack2(d[0], d[1]), pack2(d[2], d[3]), pack2(d[4], d[5]), pack2(d[6], d[7]));
            *reinterpret_cast<uint4*>(dYs + 2048 + r * 16) = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) {
                l += __shfl_xor_sync(0xffffffffu, l, m);
#pragma unroll
                for (int j = 0; j < AVBD_MLP_OUT; j++) d[j] += __shfl_xor_sync(0xffffffffu, d[j], m);
            }
            if (lane == 0) {
                atomicAdd(lsum, l / (float)(B * AVBD_MLP_OUT));
#pragma unroll
                for (int j = 0; j < AVBD_MLP_OUT; j++) atomicAdd(db + 3 * HID + j, d[j]);
            }
        }
        // dW4^T = H3^T dY, then dH3 = dY W4
        if (!run([&] { product(work, Hs[2], true, dYs, 128, true, 8, id_w4); }, nothing)) break;
        if (warp < 4) {
            float v[16];
            tc::tmem_ld16(work + trow, v);
#pragma unroll
            for (int j = 0; j < AVBD_MLP_OUT; j++) atomicAdd(G + OFF_W4 + j * HID + r, v[j]);
        }
        if (!run([&] { product(work, dYs, false, W4s, OUT, true, 1, id_hb); }, nothing)) break;
        // layer 3
        activate_grad(tmem + 256, bias + 2 * HID, Hs[2], db + 2 * HID);
        if (!run([&] {
                product(tmem + 256, Hs[2], true, Hs[1], 128, true, 8, id_w);
                product(work, Hs[2], false, W3s, HID, true, HID / 16, id_hb);
            }, nothing))
            break;
        // layer 2, layer 3's gradient flushed beside its products
        activate_grad(tmem + 128, bias + HID, Hs[1], db + HID);
        if (!run([&] {
                product(tmem + 128, Hs[1], true, Hs[0], 128, true, 8, id_w);
                product(work, Hs[1], false, W2s, HID, true, HID / 16, id_hb);
            }, [&] { flush(tmem + 256, G + OFF_W3); }))
            break;
        // layer 1
        activate_grad(tmem, bias, Hs[0], db);
        if (!run([&] { product(tmem, Hs[0], true, Xs, 128, true, 8, id_w1); }, [&] { flush(tmem + 128, G + OFF_W2); })) break;
        if (warp < 8) {  // [128][32]: warp w rows 32 (w % 4).., columns 16 (w / 4)..
            const unsigned cc = (warp >> 2) * 16;
            float v[16];
            tc::tmem_ld16(tmem + trow + cc, v);
#pragma unroll
            for (int j = 0; j < 16; j += 4)
                red_add4(G + OFF_W1 + r * IN + cc + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
    }
    if (!ok) drain_after_timeout(bar, phase);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tmem_dealloc(tmem, 512);
        tc::tmem_relinquish();
    }
    if (tid < HID) {
        atomicAdd(G + OFF_B1 + tid, db[tid]);
        atomicAdd(G + OFF_B2 + tid, db[HID + tid]);
        atomicAdd(G + OFF_B3 + tid, db[2 * HID + tid]);
    }
    if (tid < AVBD_MLP_OUT) atomicAdd(G + OFF_B4 + tid, db[3 * HID + tid]);
    if (tid == 0) {
        atomicAdd(loss, *lsum);
        if (!ok) atomicExch(err, (int)AVBD_ERR_BARRIER_TIMEOUT);
    }
}

// one master FP32 parameter into its BF16 weight or FP32 bias
AVBD_D void pack_param(unsigned i, float p, bf16* w1, bf16* w2, bf16* w3, bf16* w4, float* b) {
    if (i < OFF_B1) w1[i] = __float2bfloat16_rn(p);
    else if (i < OFF_W2) b[i - OFF_B1] = p;
    else if (i < OFF_B2) w2[i - OFF_W2] = __float2bfloat16_rn(p);
    else if (i < OFF_W3) b[HID + i - OFF_B2] = p;
    else if (i < OFF_B3) w3[i - OFF_W3] = __float2bfloat16_rn(p);
    else if (i < OFF_W4) b[2 * HID + i - OFF_B3] = p;
    else if (i < OFF_B4) w4[i - OFF_W4] = __float2bfloat16_rn(p);
    else b[3 * HID + i - OFF_B4] = p;
}

__global__ void k_pack(const float* P, bf16* w1, bf16* w2, bf16* w3, bf16* w4, float* b) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < NPAR) pack_param(i, P[i], w1, w2, w3, w4, b);
}

// padding that must stay zero: inputs 27..31 of W1, outputs 3..15 of W4 / b4
AVBD_D bool frozen(unsigned i) {
    if (i < OFF_B1) return (i % IN) >= AVBD_MLP_IN;
    if (i >= OFF_W4 && i < OFF_B4) return (i - OFF_W4) / HID >= AVBD_MLP_OUT;
    if (i >= OFF_B4) return i - OFF_B4 >= AVBD_MLP_OUT;
    return false;
}

// Adam on the master parameters, which are packed again as they change
__global__ void k_adam(float* P, const float* G, float* Mo, float* Vo, float lr, float c1, float c2, bf16* w1, bf16* w2,
                       bf16* w3, bf16* w4, float* b) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NPAR || frozen(i)) return;
    float g = G[i];
    float m = 0.9f * Mo[i] + 0.1f * g;
    float v = 0.999f * Vo[i] + 0.001f * g * g;
    Mo[i] = m;
    Vo[i] = v;
    const float p = P[i] - lr * (m / c1) / (sqrtf(v / c2) + 1e-8f);
    P[i] = p;
    pack_param(i, p, w1, w2, w3, w4, b);
}

inline unsigned nb(size_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

}  // namespace

// BF16 weights + FP32 biases of one MLP on the device
struct MlpDevice {
    bf16 *w1 = nullptr, *w2 = nullptr, *w3 = nullptr, *w4 = nullptr;
    float* b = nullptr;
    float* p32 = nullptr;
    int* err = nullptr;
    int device = 0;
    bool own_err = true;
    int upload(const float* params, cudaStream_t st);
    void release();
};

int MlpDevice::upload(const float* params, cudaStream_t st) {
    if (!params) return set_error(AVBD_ERR_INVALID_ARG, "null parameters");
    auto al = [](void** p, size_t bytes) { return cudaMalloc(p, bytes); };
    if (!w1) {
        if (al((void**)&w1, sizeof(bf16) * HID * IN) || al((void**)&w2, sizeof(bf16) * HID * HID) ||
            al((void**)&w3, sizeof(bf16) * HID * HID) || al((void**)&w4, sizeof(bf16) * OUT * HID) ||
            al((void**)&b, sizeof(float) * (3 * HID + OUT)) || al((void**)&p32, sizeof(float) * NPAR) ||
            al((void**)&err, sizeof(int)))
            return set_error(AVBD_ERR_CUDA, "MLP weight allocation failed");
        cudaMemsetAsync(err, 0, sizeof(int), st);
    }
    if (cudaMemcpyAsync(p32, params, sizeof(float) * NPAR, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return set_error(AVBD_ERR_CUDA, "MLP parameter upload failed");
    k_pack<<<nb(NPAR, 256), 256, 0, st>>>(p32, w1, w2, w3, w4, b);
    cudaError_t e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? AVBD_OK : set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
}

void MlpDevice::release() {
    for (void* p : {(void*)w1, (void*)w2, (void*)w3, (void*)w4, (void*)b, (void*)p32, own_err ? (void*)err : nullptr})
        if (p) cudaFree(p);
    w1 = w2 = w3 = w4 = nullptr;
    b = p32 = nullptr;
    err = nullptr;
}

static int grid_for(int device, unsigned n) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return (int)std::max(1u, std::min((n + 127) / 128, (unsigned)sms));
}

template <typename P, bool OUT16>
static int mlp_launch_form(const MlpDevice& m, const bf16* feat, unsigned n, const MlpSink<P>& sink, cudaStream_t st) {
    static std::atomic<uint64_t> done;  // bit d: attribute set on device d
    const uint64_t bit = 1ull << (m.device & 63);
    if (!(done.load() & bit)) {
        cudaError_t e = cudaFuncSetAttribute(k_mlp_apply<P, OUT16>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_TOTAL);
        if (e != cudaSuccess) return set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
        done.fetch_or(bit);
    }
    MlpW w{m.w1, m.w2, m.w3, m.w4, m.b};
    k_mlp_apply<P, OUT16><<<grid_for(m.device, n), GROUPS * GTHREADS, SM_TOTAL, st>>>(w, feat, n, sink, m.err);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AVBD_OK : set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
}

template <typename P>
static int mlp_launch(const MlpDevice& m, const bf16* feat, unsigned n, const MlpSink<P>& sink, cudaStream_t st) {
    if (n == 0) return AVBD_OK;
    if constexpr (sizeof(P) == 4)
        if ((uintptr_t)sink.out & 15) return mlp_launch_form<P, false>(m, feat, n, sink, st);
    return mlp_launch_form<P, true>(m, feat, n, sink, st);
}

// x0 update of the engine's warm start (rows: internal vertex of each row)
template <typename P>
int mlp_apply_state(const MlpDevice& m, const void* feat, unsigned n, typename Vec4Of<P>::T* x,
                    typename Vec4Of<P>::T* xl, typename Vec4Of<P>::T* xll, const uint8_t* flags, double scale,
                    float kappa, unsigned long long* applied, cudaStream_t st) {
    MlpSink<P> s{nullptr, x, xl, xll, flags, (P)scale, kappa, applied};
    return mlp_launch<P>(m, (const bf16*)feat, n, s, st);
}
template int mlp_apply_state<float>(const MlpDevice&, const void*, unsigned, float4*, float4*, float4*,
                                    const uint8_t*, double, float, unsigned long long*, cudaStream_t);
template int mlp_apply_state<double>(const MlpDevice&, const void*, unsigned, double4a*, double4a*, double4a*,
                                     const uint8_t*, double, float, unsigned long long*, cudaStream_t);

int mlp_device_upload(MlpDevice** m, int device, const float* params, cudaStream_t st) {
    if (!*m) {
        *m = new MlpDevice();
        (*m)->device = device;
    }
    return (*m)->upload(params, st);
}
void mlp_device_free(MlpDevice* m) {
    if (m) {
        m->release();
        delete m;
    }
}
int mlp_device_error(const MlpDevice* m, cudaStream_t st) {
    int h = 0;
    if (!m || !m->err) return AVBD_OK;
    if (cudaMemcpyAsync(&h, m->err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return set_error(AVBD_ERR_CUDA, "MLP error flag read failed");
    if (!h) return AVBD_OK;
    // the flag is cleared once reported, so the object stays usable
    if (cudaMemsetAsync(m->err, 0, sizeof(int), st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess)
        return set_error(AVBD_ERR_CUDA, "MLP error flag reset failed");
    return set_error(h, "MLP kernel: a bounded wait on the tensor-core barrier gave up; every result of that "
                        "launch is invalid");
}

}  // namespace avbd

using namespace avbd;

// ------------------------------------------------------------------- C-ABI
struct avbd_mlp {
    MlpDevice* m = nullptr;
    cudaStream_t st = nullptr;
};

struct avbd_mlp_trainer {
    int device = 0;
    unsigned B = 0;
    cudaStream_t st = nullptr;
    MlpDevice w;                  // BF16 [out][in] weights + biases
    float *G = nullptr, *Mo = nullptr, *Vo = nullptr;  // G: gradient, then the loss and the kernels' error flag
    float* status = nullptr;      // pinned host copy of the loss and the flag
    unsigned t = 0;
    std::vector<void*> allocs;
};

extern "C" {

int avbd_gemm_bf16(const void* A, unsigned lda, const void* B, unsigned ldb, float* C, unsigned ldc, unsigned M,
                   unsigned N, unsigned K, int accumulate, void* stream) {
    if (!A || !B || !C) return set_error(AVBD_ERR_INVALID_ARG, "null operand");
    int* err = nullptr;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMalloc(&err, sizeof(int)) != cudaSuccess) return set_error(AVBD_ERR_CUDA, "cudaMalloc");
    cudaMemsetAsync(err, 0, sizeof(int), st);
    int rc = gemm_bf16((const bf16*)A, lda, (const bf16*)B, ldb, C, ldc, M, N, K, accumulate != 0, st, err);
    int h = 0;
    cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    cudaFree(err);
    if (rc) return rc;
    if (e != cudaSuccess) return set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
    return h ? set_error(h, "GEMM: a bounded wait on the tensor-core barrier gave up") : AVBD_OK;
}

int avbd_debug_set_wait_limit(int device, unsigned polls) {
    int prev = 0;
    if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess)
        return set_error(AVBD_ERR_NO_DEVICE, "cudaSetDevice failed");
    cudaError_t e = cudaMemcpyToSymbol(g_wait_polls, &polls, sizeof(polls));
    int rc = e == cudaSuccess ? solve_set_wait_limit(polls) : AVBD_OK;
    if (e == cudaSuccess && rc == AVBD_OK) rc = contacts_set_wait_limit(polls);
    if (e == cudaSuccess && rc == AVBD_OK) e = cudaDeviceSynchronize();
    cudaSetDevice(prev);
    if (rc != AVBD_OK) return rc;
    return e == cudaSuccess ? AVBD_OK : set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
}

int avbd_mlp_create(avbd_mlp** out, int device, const float* params) {
    if (!out || !params) return set_error(AVBD_ERR_INVALID_ARG, "null argument");
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return set_error(AVBD_ERR_NO_DEVICE, "cudaSetDevice failed");
    avbd_mlp* m = new avbd_mlp();
    cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking);
    if (int rc = mlp_device_upload(&m->m, device, params, m->st)) {
        mlp_device_free(m->m);
        cudaStreamDestroy(m->st);
        delete m;
        return rc;
    }
    *out = m;
    return AVBD_OK;
}

int avbd_mlp_forward(avbd_mlp* m, const void* features, unsigned n, float* out, void* stream) {
    if (!m || !features || !out) return set_error(AVBD_ERR_INVALID_ARG, "null argument");
    if ((uintptr_t)features & 15) return set_error(AVBD_ERR_INVALID_ARG, "features must be 16-byte aligned");
    cudaStream_t st = stream ? (cudaStream_t)stream : m->st;
    MlpSink<float> s{out, nullptr, nullptr, nullptr, nullptr, 0.f, 0.f, nullptr};
    if (int rc = mlp_launch<float>(*m->m, (const bf16*)features, n, s, st)) return rc;
    return mlp_device_error(m->m, st);
}

int avbd_mlp_destroy(avbd_mlp* m) {
    if (!m) return AVBD_OK;
    mlp_device_free(m->m);
    if (m->st) cudaStreamDestroy(m->st);
    delete m;
    return AVBD_OK;
}

int avbd_mlp_trainer_create(avbd_mlp_trainer** out, int device, unsigned batch, const float* params) {
    if (!out || !params) return set_error(AVBD_ERR_INVALID_ARG, "null argument");
    if (batch == 0 || batch % 128) return set_error(AVBD_ERR_INVALID_ARG, "batch must be a positive multiple of 128");
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return set_error(AVBD_ERR_NO_DEVICE, "cudaSetDevice failed");
    auto* t = new avbd_mlp_trainer();
    t->device = device;
    t->B = batch;
    cudaStreamCreateWithFlags(&t->st, cudaStreamNonBlocking);
    bool bad = false;
    auto al = [&](auto** p, size_t bytes) {
        if (bad) return;
        if (cudaMalloc((void**)p, bytes) != cudaSuccess) bad = true;
        else t->allocs.push_back((void*)*p);
    };
    al(&t->G, sizeof(float) * (NPAR + 2)); al(&t->Mo, sizeof(float) * NPAR); al(&t->Vo, sizeof(float) * NPAR);
    if (!bad && cudaMallocHost((void**)&t->status, 2 * sizeof(float)) != cudaSuccess) bad = true;
    if (bad) {
        avbd_mlp_trainer_destroy(t);
        return set_error(AVBD_ERR_CUDA, "trainer allocation failed");
    }
    t->w.device = device;
    if (int rc = t->w.upload(params, t->st)) {
        avbd_mlp_trainer_destroy(t);
        return rc;
    }
    cudaMemsetAsync(t->Mo, 0, sizeof(float) * NPAR, t->st);
    cudaMemsetAsync(t->Vo, 0, sizeof(float) * NPAR, t->st);
    // the flag lies behind the loss, so that one copy reads both
    cudaFree(t->w.err);
    t->w.err = reinterpret_cast<int*>(t->G + NPAR + 1);
    t->w.own_err = false;
    cudaMemsetAsync(t->G, 0, sizeof(float) * (NPAR + 2), t->st);
    cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_TOTAL);
    if (cudaStreamSynchronize(t->st) != cudaSuccess) {
        avbd_mlp_trainer_destroy(t);
        return set_error(AVBD_ERR_CUDA, "trainer initialisation failed");
    }
    *out = t;
    return AVBD_OK;
}

// forward + backward of one mini-batch into t->G (and the loss behind it)
static int trainer_fwd_bwd(avbd_mlp_trainer* t, const bf16* X, const float* T) {
    cudaMemsetAsync(t->G, 0, sizeof(float) * (NPAR + 1), t->st);
    const MlpW w{t->w.w1, t->w.w2, t->w.w3, t->w.w4, t->w.b};
    k_train<<<grid_for(t->device, t->B), 512, TR_TOTAL, t->st>>>(w, X, T, t->B, t->G, t->G + NPAR, t->w.err);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AVBD_OK : set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
}

// waits for the stream and reads the loss and the error flag
static int trainer_status(avbd_mlp_trainer* t, float* loss) {
    cudaMemcpyAsync(t->status, t->G + NPAR, 2 * sizeof(float), cudaMemcpyDeviceToHost, t->st);
    if (cudaStreamSynchronize(t->st) != cudaSuccess) return set_error(AVBD_ERR_CUDA, "trainer sync failed");
    if (loss) *loss = t->status[0];
    int flag;
    std::memcpy(&flag, t->status + 1, sizeof(flag));
    return flag ? mlp_device_error(&t->w, t->st) : AVBD_OK;
}

static int trainer_args(avbd_mlp_trainer* t, const void* features, const float* targets) {
    if (!t || !features || !targets) return set_error(AVBD_ERR_INVALID_ARG, "null argument");
    if ((uintptr_t)features & 15) return set_error(AVBD_ERR_INVALID_ARG, "features must be 16-byte aligned");
    return AVBD_OK;
}

int avbd_mlp_trainer_grad(avbd_mlp_trainer* t, const void* features, const float* targets, float* loss, float* grad) {
    if (int rc = trainer_args(t, features, targets)) return rc;
    if (int rc = trainer_fwd_bwd(t, (const bf16*)features, targets)) return rc;
    if (grad) cudaMemcpyAsync(grad, t->G, sizeof(float) * NPAR, cudaMemcpyDeviceToHost, t->st);
    return trainer_status(t, loss);
}

int avbd_mlp_trainer_step(avbd_mlp_trainer* t, const void* features, const float* targets, float lr, float* loss) {
    if (int rc = trainer_args(t, features, targets)) return rc;
    if (int rc = trainer_fwd_bwd(t, (const bf16*)features, targets)) return rc;
    t->t++;
    const float c1 = 1.0f - powf(0.9f, (float)t->t), c2 = 1.0f - powf(0.999f, (float)t->t);
    k_adam<<<nb(NPAR, 256), 256, 0, t->st>>>(t->w.p32, t->G, t->Mo, t->Vo, lr, c1, c2, t->w.w1, t->w.w2, t->w.w3,
                                             t->w.w4, t->w.b);
    if (loss) return trainer_status(t, loss);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AVBD_OK : set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
}

int avbd_mlp_trainer_get_params(avbd_mlp_trainer* t, float* params) {
    if (!t || !params) return set_error(AVBD_ERR_INVALID_ARG, "null argument");
    cudaMemcpyAsync(params, t->w.p32, sizeof(float) * NPAR, cudaMemcpyDeviceToHost, t->st);
    if (cudaStreamSynchronize(t->st) != cudaSuccess) return set_error(AVBD_ERR_CUDA, "trainer sync failed");
    return mlp_device_error(&t->w, t->st);
}

int avbd_mlp_trainer_destroy(avbd_mlp_trainer* t) {
    if (!t) return AVBD_OK;
    if (t->st) cudaStreamSynchronize(t->st);
    for (void* p : t->allocs) cudaFree(p);
    if (t->status) cudaFreeHost(t->status);
    t->w.release();
    if (t->st) cudaStreamDestroy(t->st);
    delete t;
    return AVBD_OK;
}

}  // extern "C"
