// solve.cu -- per-step kernels of the AVBD solve for positional (3-DOF)
// vertices: step-start energy hooks + inertial prediction, the per-color
// vertex block solve over NeoHookean tets and ground contact, Chebyshev
// acceleration fused with the contact dual update, the velocity update and
// the residual reduction.
//
// Reference behaviour followed:
//   VBDSolver::solve_Parallel step schedule     simulation/VBDSolver.hpp:48-103
//   _particleInertialUpdate                      simulation/VBDSolver.hpp:208-248
//   _solveParticle<3>                            simulation/VBDSolver.hpp:285-511
//   _particleChebyshevAcceleration               simulation/VBDSolver.hpp:513-536
//   _particleVelocityUpdate                      simulation/VBDSolver.hpp:538-566
//   NeoHookeanEnergySolver::accumulate           energy/elastic/NeoHookeanEnergySolver.hpp:121-227
//   NeoHookeanEnergySolver::updateAfterTimeStep  energy/elastic/NeoHookeanEnergySolver.hpp:70-90
//   CollisionConstraintEnergySolver (ground)     energy/collision/CollisionConstraintEnergySolver.hpp:60-285
//   GroundCollisionEnergySolver                  energy/collision/GroundCollisionEnergySolver.hpp:14-91
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "engine.h"
#include "contact_dyn.cuh"

namespace avbd {

template <typename R>
struct Consts {
    R dt, inv_dt, inv_dt2, g, kappa_max;
};

template <typename R>
static Consts<R> mkc(const StepConsts& k) {
    return Consts<R>{(R)k.dt, (R)(1.0 / k.dt), (R)(1.0 / (k.dt * k.dt)), (R)k.g, (R)k.kappa_max};
}

static inline unsigned nblocks(unsigned n, unsigned per) { return (n + per - 1) / per; }
static constexpr unsigned ITER_WARPS_MIN = 4;  // warps of work per block of an iteration launch, at least

// ----------------------------------------------------------- step start
// Energy hooks of the step start for per-vertex ground contact
// (GroundCollisionEnergySolver::updateContactPoints + CollisionConstraintEnergySolver::
// updateAfterTimeStep) followed by the inertial prediction with adaptive
// initialisation.  Both read the positions at the start of the step; the hook
// runs first, as in the reference (VBDSolver.hpp:54-62).
template <typename R>
__global__ void __launch_bounds__(256) k_begin_step(DevState<R> s, Consts<R> c) {
    unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n) return;
    using V4 = typename Vec4Of<R>::T;
    uint8_t fl = s.flags[p];
    V4 x4 = s.x[p];
    if (fl & VF_GROUND) {
        V4 k = s.gk[p], lam = s.glam[p], cp = s.gcp[p];
        uint8_t gf = s.gflag[p];
        cp.x = x4.x;
        cp.y = x4.z;
        if (lam.x > R(0)) lam.w = -x4.y;
        if ((gf & GF_UNCLAMPED) && !(gf & GF_USE_STATIC)) gf |= GF_USE_STATIC;
        lam.x *= R(AVBD_ALPHA * AVBD_GAMMA);
        lam.y *= R(AVBD_GAMMA);
        lam.z *= R(AVBD_GAMMA);
        R gk;
        gk = R(AVBD_GAMMA) * k.x; k.x = (gk < k.w) ? k.w : gk;
        gk = R(AVBD_GAMMA) * k.y; k.y = (gk < k.w) ? k.w : gk;
        gk = R(AVBD_GAMMA) * k.z; k.z = (gk < k.w) ? k.w : gk;
        s.gk[p] = k;
        s.glam[p] = lam;
        s.gcp[p] = cp;
        s.gflag[p] = gf;
    }
    if (fl & (VF_FIXED | VF_ORIENTED)) return;
    V3<R> x = xyz(x4);
    V3<R> v = xyz(s.v[p]), vp = xyz(s.vp[p]);
    V3<R> a = c.inv_dt * (v - vp);
    V3<R> aext = mk3<R>(0, -c.g, 0);
    R an = c.g;
    R t = 0;
    if (an > R(1e-12)) {
        R al = dot3(a, aext) / an;
        if (al > an) t = 1;
        else if (al < R(0)) t = 0;
        else t = al / an;
    }
    V3<R> at = t * aext;
    R dt2 = c.dt * c.dt;
    V3<R> y = (x + c.dt * v) + dt2 * aext;
    V3<R> xn = x + (c.dt * v + dt2 * at);
    V4 y4 = s.y[p];
    s.y[p] = make4<R>(y, y4.w);
    V4 o = make4<R>(xn, x4.w);
    s.x[p] = o;
    s.xl[p] = o;
    s.xll[p] = o;
}

// E_prev = 1/2 (F_prev^T F_prev - I) of every tet from the previous positions
// (NeoHookeanEnergySolver::updateAfterTimeStep).  Only run when some tet has
// strain-rate damping; without damping E_prev is never read.
template <typename R>
__global__ void __launch_bounds__(256) k_tet_eprev(DevState<R> s) {
    unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= s.ntets) return;
    uint4 id = s.tet_idx[t];
    V3<R> x0 = xyz(s.xp[id.x]), x1 = xyz(s.xp[id.y]), x2 = xyz(s.xp[id.z]), x3 = xyz(s.xp[id.w]);
    V3<R> q0 = xyz(s.tet_q[3 * t]), q1 = xyz(s.tet_q[3 * t + 1]), q2 = xyz(s.tet_q[3 * t + 2]);
    V3<R> a = x0 - x3, b = x1 - x3, d = x2 - x3;
    // F = [a b d] Q: column j = a Q0j + b Q1j + d Q2j
    V3<R> F0 = q0.x * a + q1.x * b + q2.x * d;
    V3<R> F1 = q0.y * a + q1.y * b + q2.y * d;
    V3<R> F2 = q0.z * a + q1.z * b + q2.z * d;
    typename Vec4Of<R>::T e0, e1 = s.tet_e[2 * t + 1];
    e0.x = R(0.5) * (dot3(F0, F0) - R(1));
    e0.y = R(0.5) * (dot3(F1, F1) - R(1));
    e0.z = R(0.5) * (dot3(F2, F2) - R(1));
    e0.w = R(0.5) * dot3(F0, F1);
    e1.x = R(0.5) * dot3(F0, F2);
    e1.y = R(0.5) * dot3(F1, F2);
    s.tet_e[2 * t] = e0;
    s.tet_e[2 * t + 1] = e1;
}

// ------------------------------------------------------- vertex block
template <typename R>
AVBD_D IncRec<R> load_rec(const IncRec<R>* p);

template <>
AVBD_D IncRec<float> load_rec<float>(const IncRec<float>* p) {
    const float4* q = reinterpret_cast<const float4*>(p);
    float4 a = __ldcs(q), b = __ldcs(q + 1), c = __ldcs(q + 2), d = __ldcs(q + 3);
    IncRec<float> r;
    r.o[0] = __float_as_uint(a.x); r.o[1] = __float_as_uint(a.y); r.o[2] = __float_as_uint(a.z);
    r.tet = __float_as_uint(a.w);
    r.d[0] = b.x; r.d[1] = b.y; r.d[2] = b.z; r.d[3] = b.w;
    r.d[4] = c.x; r.d[5] = c.y; r.d[6] = c.z; r.d[7] = c.w;
    r.d[8] = d.x; r.vlam = d.y; r.vmu = d.z; r.mol = d.w;
    return r;
}
AVBD_D void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
AVBD_D void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

template <>
AVBD_D IncRec<double> load_rec<double>(const IncRec<double>* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const uint4 h = __ldcs(reinterpret_cast<const uint4*>(p));
    IncRec<double> r;
    r.o[0] = h.x; r.o[1] = h.y; r.o[2] = h.z; r.tet = h.w;
    double2 v;
    v = __ldcs(q + 1); r.d[0] = v.x; r.d[1] = v.y;
    v = __ldcs(q + 2); r.d[2] = v.x; r.d[3] = v.y;
    v = __ldcs(q + 3); r.d[4] = v.x; r.d[5] = v.y;
    v = __ldcs(q + 4); r.d[6] = v.x; r.d[7] = v.y;
    v = __ldcs(q + 5); r.d[8] = v.x; r.vlam = v.y;
    v = __ldcs(q + 6); r.vmu = v.x; r.mol = v.y;
    return r;
}

// Accumulated block: gradient in the state precision P, Hessian in HT.  The
// Hessian only shapes the Newton step, never the converged state, so the
// mixed mode keeps it in FP32 while the gradient (which the residual
// measures) is formed in FP64.
template <typename P, typename HT>
struct Block3 {
    P g0 = 0, g1 = 0, g2 = 0;
    HT h00 = 0, h11 = 0, h22 = 0, h01 = 0, h02 = 0, h12 = 0;
};

// One NeoHookean incidence: NeoHookeanEnergySolver::accumulate with the tet
// restated relative to the solved vertex (see IncRec).  P is the precision of
// positions and gradient, RS the stored record scalar, HT the Hessian type.
// The terms from the three edge vectors e_j = x_(o_j) - x_i; `tet` indexes
// the damping state.
template <typename P, typename RS, typename HT, bool DAMP, typename RD>
AVBD_D void accumulate_tet_e(const DevState<P>& s, const RD& r, unsigned tet, V3<P> e1, V3<P> e2, V3<P> e3, P dt,
                             Block3<P, HT>& B) {
    V3<P> d1 = mk3<P>(r.d[0], r.d[1], r.d[2]);
    V3<P> d2 = mk3<P>(r.d[3], r.d[4], r.d[5]);
    V3<P> d3 = mk3<P>(r.d[6], r.d[7], r.d[8]);
    V3<P> dw = mk3<P>(-(d1.x + d2.x + d3.x), -(d1.y + d2.y + d3.y), -(d1.z + d2.z + d3.z));
    // columns of F
    V3<P> F0 = d1.x * e1 + d2.x * e2 + d3.x * e3;
    V3<P> F1 = d1.y * e1 + d2.y * e2 + d3.y * e3;
    V3<P> F2 = d1.z * e1 + d2.z * e2 + d3.z * e3;
    V3<P> c0 = cross3(F1, F2), c1 = cross3(F2, F0), c2 = cross3(F0, F1);
    P J = dot3(F0, c0);
    V3<P> Fc = dw.x * c0 + dw.y * c1 + dw.z * c2;   // cof(F) d
    V3<P> Fd = dw.x * F0 + dw.y * F1 + dw.z * F2;   // F d
    P hyd = (P)r.vlam * ((J - P(1)) - (P)r.mol);     // V lambda (J - mu/lambda - 1)
    P dev = (P)r.vmu;
    P qn2 = dot3(dw, dw);
    B.g0 += hyd * Fc.x + dev * Fd.x;
    B.g1 += hyd * Fc.y + dev * Fd.y;
    B.g2 += hyd * Fc.z + dev * Fd.z;
    const HT vl = (HT)r.vlam, fx = (HT)Fc.x, fy = (HT)Fc.y, fz = (HT)Fc.z;
    const HT dg = (HT)(dev * qn2);
    B.h00 += vl * fx * fx + dg;
    B.h11 += vl * fy * fy + dg;
    B.h22 += vl * fz * fz + dg;
    B.h01 += vl * fx * fy;
    B.h02 += vl * fx * fz;
    B.h12 += vl * fy * fz;
    if constexpr (DAMP) {
        typename Vec4Of<P>::T e0 = s.tet_e[2 * tet], e1v = s.tet_e[2 * tet + 1];
        P vkd = e1v.z;
        if (vkd != P(0)) {
            P idt = P(1) / dt;
            // Edot = (1/2 (F^T F - I) - E_prev) / dt
            P E00 = (P(0.5) * (dot3(F0, F0) - P(1)) - e0.x) * idt;
            P E11 = (P(0.5) * (dot3(F1, F1) - P(1)) - e0.y) * idt;
            P E22 = (P(0.5) * (dot3(F2, F2) - P(1)) - e0.z) * idt;
            P E01 = (P(0.5) * dot3(F0, F1) - e0.w) * idt;
            P E02 = (P(0.5) * dot3(F0, F2) - e1v.x) * idt;
            P E12 = (P(0.5) * dot3(F1, F2) - e1v.y) * idt;
            V3<P> Ed = mk3<P>(E00 * dw.x + E01 * dw.y + E02 * dw.z, E01 * dw.x + E11 * dw.y + E12 * dw.z,
                              E02 * dw.x + E12 * dw.y + E22 * dw.z);
            P damp = P(2) * idt * vkd;
            V3<P> FEd = Ed.x * F0 + Ed.y * F1 + Ed.z * F2;
            B.g0 += damp * FEd.x;
            B.g1 += damp * FEd.y;
            B.g2 += damp * FEd.z;
            HT diag = (HT)(damp * dot3(dw, Ed));
            HT al = (HT)(P(0.5) * damp * idt);
            HT q2 = (HT)qn2;
            // F F^T = sum_c F_c F_c^T
            HT f00 = (HT)(F0.x * F0.x + F1.x * F1.x + F2.x * F2.x);
            HT f11 = (HT)(F0.y * F0.y + F1.y * F1.y + F2.y * F2.y);
            HT f22 = (HT)(F0.z * F0.z + F1.z * F1.z + F2.z * F2.z);
            HT f01 = (HT)(F0.x * F0.y + F1.x * F1.y + F2.x * F2.y);
            HT f02 = (HT)(F0.x * F0.z + F1.x * F1.z + F2.x * F2.z);
            HT f12 = (HT)(F0.y * F0.z + F1.y * F1.z + F2.y * F2.z);
            HT dx = (HT)Fd.x, dy = (HT)Fd.y, dz = (HT)Fd.z;
            B.h00 += diag + al * (f00 * q2 + dx * dx);
            B.h11 += diag + al * (f11 * q2 + dy * dy);
            B.h22 += diag + al * (f22 * q2 + dz * dz);
            B.h01 += al * (f01 * q2 + dx * dy);
            B.h02 += al * (f02 * q2 + dx * dz);
            B.h12 += al * (f12 * q2 + dy * dz);
        }
    }
}

// COH: neighbour positions by coherent loads (k_iterate, whose own
// launch writes them); otherwise through the read-only path.
template <typename P, typename RS, typename HT, bool DAMP, bool COH = false>
AVBD_D void accumulate_tet(const DevState<P>& s, const IncRec<RS>& r, V3<P> xi, P dt, Block3<P, HT>& B) {
    V3<P> e1, e2, e3;
    if constexpr (COH) {
        e1 = xyz(s.x[r.o[0]]) - xi;
        e2 = xyz(s.x[r.o[1]]) - xi;
        e3 = xyz(s.x[r.o[2]]) - xi;
    } else {
        e1 = xyz(ld_ro(s.x + r.o[0])) - xi;
        e2 = xyz(ld_ro(s.x + r.o[1])) - xi;
        e3 = xyz(ld_ro(s.x + r.o[2])) - xi;
    }
    accumulate_tet_e<P, RS, HT, DAMP>(s, r, r.tet, e1, e2, e3, dt, B);
}

// Loads of the star form: read once per launch, so kept out of L1, where the
// neighbour gathers live.
AVBD_D uint2 ld_once(const uint2* p) {
    uint2 v;
    asm("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
AVBD_D uint32_t ld_once(const uint32_t* p) {
    uint32_t v;
    asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
AVBD_D StarNb<float> ld_once(const StarNb<float>* p) {
    const uint2 v = ld_once(reinterpret_cast<const uint2*>(p));
    return {v.x, __uint_as_float(v.y)};
}
AVBD_D StarTet<float> ld_once(const StarTet<float>* p) {
    const uint2 v = ld_once(reinterpret_cast<const uint2*>(p));
    return {__uint_as_float(v.x), __uint_as_float(v.y)};
}
AVBD_D StarNb<double> ld_once(const StarNb<double>* p) {
    StarNb<double> v;
    asm("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.idx), "=r"(v.pad) : "l"(p));
    asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v.w) : "l"(&p->w));
    return v;
}
AVBD_D StarTet<double> ld_once(const StarTet<double>* p) {
    StarTet<double> v;
    asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.a), "=d"(v.r) : "l"(p));
    return v;
}

// Shared-memory staging of the neighbour edges: component c of edge j of the
// block's vertex slot g lies at [(c max_nb + j) stride + g].  Lanes of one
// vertex read different j and neighbouring vertices mostly the same j, so the
// stride is skewed by a half-warp's (FP64) or a warp's (FP32) width over
// LANES to spread both over the banks.
template <typename P, int LANES, int THREADS = 256>
struct StarStage {
    static constexpr unsigned GROUPS = THREADS / LANES;
    static constexpr unsigned STRIDE = GROUPS + (sizeof(P) == 8 ? 16 : 32) / LANES;
    static unsigned bytes(unsigned max_nb) { return 3 * max_nb * STRIDE * (unsigned)sizeof(P); }
};

// double of a float whose magnitude is normal or zero (element constants, see
// build_star), by integer arithmetic: the mantissa moves up 29 bits and the
// exponent's bias grows by 896.  The conversion instruction runs on a unit of
// a few lanes (at one conversion per constant it was the busiest pipe of the
// mixed solve); zero becomes 2^-127, which vanishes next to any element.
AVBD_D double widen(float f) {
    const uint32_t u = __float_as_uint(f);
    const unsigned long long m = (unsigned long long)(u & 0x7FFFFFFFu) * 0x20000000ull + 0x3800000000000000ull;
    return __hiloint2double((int)((uint32_t)(m >> 32) | (u & 0x80000000u)), (int)(uint32_t)m);
}
template <typename P> AVBD_D P const_as(float f) { return (P)f; }
template <> AVBD_D double const_as<double>(float f) { return widen(f); }
template <typename P> AVBD_D P const_as(double f) { return (P)f; }

// One tet of the star form: its edges from the staging slot.
template <typename P, typename RS, typename HT, unsigned ST>
AVBD_D void star_tet(const StarTet<RS>& q, uint32_t l, const P* es, unsigned K, Block3<P, HT>& B) {
    const P* p1 = es + (l & 255u) * ST;
    const P* p2 = es + (l >> 8 & 255u) * ST;
    const P* p3 = es + (l >> 16) * ST;
    const V3<P> e1 = mk3(p1[0], p1[K * ST], p1[2 * K * ST]);
    const V3<P> f2 = mk3(p2[0], p2[K * ST], p2[2 * K * ST]) - e1;
    const V3<P> f3 = mk3(p3[0], p3[K * ST], p3[2 * K * ST]) - e1;
    const V3<P> N = cross3(f2, f3);
    const P qa = const_as<P>(q.a);
    const P h = qa * (const_as<P>(q.r) - dot3(e1, N));
    B.g0 += h * N.x;
    B.g1 += h * N.y;
    B.g2 += h * N.z;
    const HT nx = (HT)N.x, ny = (HT)N.y, nz = (HT)N.z, a = (HT)qa;
    const HT ax = a * nx, ay = a * ny, az = a * nz;
    B.h00 += ax * nx;
    B.h11 += ay * ny;
    B.h22 += az * nz;
    B.h01 += ax * ny;
    B.h02 += ax * nz;
    B.h12 += ay * nz;
}

// One neighbour of the star form: its edge staged, its weight applied.
template <typename P, typename RS, typename HT, unsigned ST>
AVBD_D void star_edge(RS wr, V3<P> e, P* d, unsigned K, Block3<P, HT>& B) {
    d[0] = e.x;
    d[K * ST] = e.y;
    d[2 * K * ST] = e.z;
    const P w = const_as<P>(wr);
    B.g0 += w * e.x;
    B.g1 += w * e.y;
    B.g2 += w * e.z;
}

// The block of a vertex from its star form (StarNb): the edges to the distinct
// neighbours are gathered once (14 instead of 61 positions on the split hex
// grids) and staged in shared memory, the deviatoric part summed over them;
// then each tet takes its three edges from there.  es: this vertex's slot.
template <typename P, typename RS, typename HT, int LANES, bool COH, int THREADS>
AVBD_D void accumulate_star(const DevState<P>& s, const TetElems<RS>& el, uint2 o0, uint2 o1, unsigned lane, V3<P> xi,
                            P* es, Block3<P, HT>& B) {
    constexpr unsigned ST = StarStage<P, LANES, THREADS>::STRIDE;
    constexpr unsigned U = LANES <= 2 ? 4 : 2;  // neighbour gathers in flight per lane
    const unsigned K = el.max_nb, n = s.n;
    auto plain = [n](unsigned idx) { return idx < n ? idx : idx - n; };  // of a tagged id (StarNb)
    for (unsigned j = o0.x + lane; j < o1.x; j += U * LANES) {
        StarNb<RS> q[U];
        V3<P> e[U];
#pragma unroll
        for (unsigned u = 0; u < U; u++)
            if (j + u * LANES < o1.x) q[u] = ld_once(el.nb + j + u * LANES);
#pragma unroll
        for (unsigned u = 0; u < U; u++)
            if (j + u * LANES < o1.x) e[u] = xyz(COH ? s.x[plain(q[u].idx)] : ld_ro(s.x + plain(q[u].idx)));
#pragma unroll
        for (unsigned u = 0; u < U; u++)
            if (j + u * LANES < o1.x)
                star_edge<P, RS, HT, ST>(q[u].w, e[u] - xi, es + (j + u * LANES - o0.x) * ST, K, B);
    }
    __syncwarp();
#pragma unroll 2
    for (unsigned t = o0.y + lane; t < o1.y; t += LANES) {
        const StarTet<RS> q = ld_once(el.tet + t);
        star_tet<P, RS, HT, ST>(q, ld_once(el.loc + t), es, K, B);
    }
    __syncwarp();  // the slot is refilled for the lane group's next vertex
}

// Ground contact term of the block (CollisionConstraintEnergySolver::accumulate<3>
// with GroundCollisionConstraintSolver): the Hessian k grad C grad C^T is always
// added, the gradient is gated by the clamped multipliers.
template <typename P, typename HT>
AVBD_D void accumulate_ground(typename Vec4Of<P>::T k, typename Vec4Of<P>::T lam, typename Vec4Of<P>::T cp, uint8_t gf,
                              V3<P> xi, Block3<P, HT>& B) {
    P Cn = -xi.y, Ct = xi.x - cp.x, Cb = xi.z - cp.y;
    P cc = Cn - P(AVBD_ALPHA) * lam.w;
    P ln = k.x * cc + lam.x;
    if (ln > P(0)) {  // out of contact the Coulomb cone is a point: no force
        P lt = k.y * Ct + lam.y, lb = k.z * Cb + lam.z;
        P mag = sqrt(lt * lt + lb * lb);
        P mu = (gf & GF_USE_STATIC) ? cp.z : cp.w;
        P mx = mu * ln;
        if (mag > mx) {
            P sc = mx / (mag + P(1e-8));
            lt = lt * sc;
            lb = lb * sc;
        }
        B.g0 += lt;
        B.g1 += -ln;
        B.g2 += lb;
    }
    B.h00 += (HT)k.y;
    B.h11 += (HT)k.x;
    B.h22 += (HT)k.z;
}

template <int LANES, typename P, typename HT>
AVBD_D void reduce_block(Block3<P, HT>& B) {
#pragma unroll
    for (int m = LANES / 2; m >= 1; m >>= 1) {
        B.g0 += shfl_xor(B.g0, m);
        B.g1 += shfl_xor(B.g1, m);
        B.g2 += shfl_xor(B.g2, m);
        B.h00 += shfl_xor(B.h00, m);
        B.h11 += shfl_xor(B.h11, m);
        B.h22 += shfl_xor(B.h22, m);
        B.h01 += shfl_xor(B.h01, m);
        B.h02 += shfl_xor(B.h02, m);
        B.h12 += shfl_xor(B.h12, m);
    }
}

enum { MODE_SOLVE = 0, MODE_RESIDUAL = 1, MODE_DEBUG = 2, MODE_FEATURES = 3 };

// FP64 solve of a block above the condition threshold; counted.
template <typename P>
__device__ __noinline__ V3<P> solve_block_d(Sym3<P> A, V3<P> rhs, unsigned long long* counters) {
    double M[3][3] = {{(double)A.a00, (double)A.a01, (double)A.a02},
                      {(double)A.a01, (double)A.a11, (double)A.a12},
                      {(double)A.a02, (double)A.a12, (double)A.a22}};
    double bb[3] = {(double)rhs.x, (double)rhs.y, (double)rhs.z}, xx[3];
    lu_solve_d<3>(M, bb, xx);
    atomicAdd(counters, 1ull);
    return mk3<P>((P)xx[0], (P)xx[1], (P)xx[2]);
}


// Vertex block solve of one color slab: LANES threads per vertex stream the
// vertex's incidence records, each lane accumulating its tets, then a shuffle
// reduction and the 3x3 solve by the group's first lane.  MODE_RESIDUAL
// evaluates |m/h^2 (x-y) + grad| instead of updating; MODE_DEBUG exports the
// accumulated block; MODE_FEATURES writes the learned warm start's 32 BF16
// input features of the vertex (row p of `out`) at the current iterate.
// Resident blocks of 256 threads asked of the compiler: the mixed mode
// (double state, float records) would take 92 registers (2 blocks per SM);
// at 3 blocks (80 registers, ~100 bytes of spill) its vertex solve ran 15 %
// faster over a whole run-to-tolerance step of the 1024-cube batch.  FP32
// fits 4 blocks (64 registers) without spills; FP64 keeps the default.
template <typename P, typename RS, int FORM>
struct SolveMinBlocks {
    static constexpr int value = FORM == 0 ? (sizeof(P) == 4 ? 4 : 3) : sizeof(P) == 4 ? 4 : (sizeof(RS) == 4 ? 3 : 1);
};

// DYN: the instantiation for vertices with dynamic contact energies or a
// color changed by the recoloring, launched over per-color lists; the slab
// launches (DYN false) skip those vertices and carry no dynamic code.
// FORM: the element data the context holds -- the star form, or the records
// without or with damping.
enum ElemForm { FORM_STAR = 0, FORM_REC = 1, FORM_DAMP = 2 };

template <typename P, typename RS, typename HT, int LANES, int FORM, bool GROUND, int MODE, bool DYN, bool COH = false,
          int THREADS = 256>
__device__ __forceinline__ void tet_vertex(const DevState<P>& s, const TetElems<RS>& el, unsigned begin,
                                           unsigned count, unsigned gi, unsigned lane, const Consts<P>& c,
                                           unsigned long long* counters, double* out, const SceneTol& T,
                                           const float4* __restrict__ aux, const uint32_t* __restrict__ list,
                                           double* acc = nullptr) {
    bool active = gi < count;
    unsigned p = list ? (active ? list[gi] : 0u) : begin + (active ? gi : 0);
    uint8_t fl = active ? s.flags[p] : 0;
    if (MODE != MODE_SOLVE && (fl & (VF_FIXED | VF_ORIENTED))) active = false;
    // vertices with dynamic contacts or a new color are solved from their color's list
    if ((MODE == MODE_SOLVE || MODE == MODE_RESIDUAL) && !DYN && s.dyn_skip && active && s.dyn_skip[p])
        active = false;
    // per-scene run-to-tolerance: converged scenes are skipped before any record is read
    if (MODE == MODE_SOLVE && T.active && active && !T.active[T.scene[p]]) active = false;
    if (MODE == MODE_RESIDUAL && T.cand && active && !T.cand[T.scene[p]]) active = false;
    Block3<P, HT> B;
    V3<P> xi = mk3<P>(0, 0, 0);
    // MODE_FEATURES: sum of the other vertices' velocities and of mu/lambda over the incident tets
    float fv0 = 0.f, fv1 = 0.f, fv2 = 0.f, fmol = 0.f, fcnt = 0.f;
    if constexpr (FORM == FORM_STAR) {
        extern __shared__ __align__(16) unsigned char stage[];
        P* es = reinterpret_cast<P*>(stage) + threadIdx.x / LANES;
        uint2 o0 = make_uint2(0, 0), o1 = o0;
        if (active) {
            xi = xyz(s.x[p]);
            o0 = el.star[p];
            o1 = el.star[p + 1];
        }
        accumulate_star<P, RS, HT, LANES, COH, THREADS>(s, el, o0, o1, lane, xi, es, B);
        if (active && lane == 0) {
            const HT hd = (HT)el.hd[p];
            B.h00 += hd;
            B.h11 += hd;
            B.h22 += hd;
        }
        if constexpr (MODE == MODE_FEATURES) {
            for (unsigned t = o0.y + lane; t < o1.y; t += LANES) {
                const uint32_t l = el.loc[t];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const unsigned o = el.nb[o0.x + (l >> 8 * j & 255u)].idx;
                    typename Vec4Of<P>::T vo = s.v[o < s.n ? o : o - s.n];
                    fv0 += (float)vo.x;
                    fv1 += (float)vo.y;
                    fv2 += (float)vo.z;
                }
                fcnt += 1.f;
            }
            if (active && lane == 0) fmol = el.mol[p];
        }
    } else if (active) {
        xi = xyz(s.x[p]);
        const IncRec<RS>* __restrict__ inc = el.inc;
        unsigned b = el.inc_begin[p], e = el.inc_begin[p + 1];
        // the next record is fetched into L1 while this one is processed (a
        // register copy of it, as a software pipeline, spilled: 192 B of
        // spill in the mixed mode at 3 blocks per SM, 3 % slower), and the
        // record three further on into L2
        unsigned k = b + lane;
        while (k < e) {
            const unsigned kn = k + LANES;
            if (kn < e) prefetch_l1(inc + kn);
            IncRec<RS> r = load_rec<RS>(inc + k);
            if (kn + 3 * LANES < e) prefetch_l2(inc + kn + 3 * LANES);
            accumulate_tet<P, RS, HT, FORM == FORM_DAMP, COH>(s, r, xi, c.dt, B);
            if constexpr (MODE == MODE_FEATURES) {
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    typename Vec4Of<P>::T vo = s.v[r.o[j]];
                    fv0 += (float)vo.x;
                    fv1 += (float)vo.y;
                    fv2 += (float)vo.z;
                }
                fmol += (float)r.mol;
                fcnt += 1.f;
            }
            k = kn;
        }
    }
    if constexpr (DYN) {
        // dynamic energies (VBDSolver.hpp:397-446): triangle-rigid then
        // triangle-rod contacts, each in slot order, spread over the lanes
        // (a contact term is a chain of rotation and Jacobian functions)
        if (active) {
            const unsigned e = s.dyn_begin[p + 1];
            for (unsigned k = s.dyn_begin[p] + lane; k < e; k += LANES) {
                const uint32_t en = s.dyn_ent[k];
                dyn_accumulate3<P, HT>(s, dyn_pool(en), dyn_slot(en), dyn_local(en), B);
            }
        }
    }
    reduce_block<LANES>(B);
    if constexpr (MODE == MODE_FEATURES) {
#pragma unroll
        for (int m = LANES / 2; m >= 1; m >>= 1) {
            fv0 += shfl_xor(fv0, m);
            fv1 += shfl_xor(fv1, m);
            fv2 += shfl_xor(fv2, m);
            fmol += shfl_xor(fmol, m);
            fcnt += shfl_xor(fcnt, m);
        }
    }
    if (!active || lane != 0) {
        if constexpr (MODE == MODE_RESIDUAL) {
            // keep the warp reduction below well defined
        } else {
            return;
        }
    }
    double r2 = 0.0, mg2 = 0.0;
    if (active && lane == 0) {
        if (GROUND && (fl & VF_GROUND))
            accumulate_ground<P, HT>(s.gk[p], s.glam[p], s.gcp[p], s.gflag[p], xi, B);
        typename Vec4Of<P>::T y4 = s.y[p];
        P m = y4.w;
        P cm = m * c.inv_dt2;
        V3<P> d = xi - xyz(y4);
        if constexpr (MODE == MODE_SOLVE) {
            Sym3<P> A{cm + (P)B.h00, cm + (P)B.h11, cm + (P)B.h22, (P)B.h01, (P)B.h02, (P)B.h12};
            V3<P> rhs = mk3<P>(-cm * d.x - B.g0, -cm * d.y - B.g1, -cm * d.z - B.g2);
            if (T.r2) {  // in-sweep residual: the block RHS just before this vertex's update
                double q = (double)rhs.x * (double)rhs.x + (double)rhs.y * (double)rhs.y +
                           (double)rhs.z * (double)rhs.z;
                if (acc) *acc += q;  // one scene per block: summed over the block
                else atomicAdd(T.r2 + T.scene[p], q);
            }
            V3<P> dx;
            if (!solve_sym3<P>(A, rhs, c.kappa_max, dx)) dx = solve_block_d(A, rhs, counters);
            typename Vec4Of<P>::T o = make4<P>(xi + dx, P(0));
            // an intra-color conflict buffers the update (VBDSolver.hpp:505-509)
            if (DYN && s.conflicted[p]) s.buffered[p] = o;
            else s.x[p] = o;
        } else if constexpr (MODE == MODE_FEATURES) {
            // feature layout of avbd_warmstart_sample (include/avbd.h)
            Sym3<P> A{cm + (P)B.h00, cm + (P)B.h11, cm + (P)B.h22, (P)B.h01, (P)B.h02, (P)B.h12};
            V3<P> rhs = mk3<P>(-cm * d.x - B.g0, -cm * d.y - B.g1, -cm * d.z - B.g2);
            V3<P> dx;
            solve_sym3<P>(A, rhs, c.kappa_max, dx);
            const float sc = 1.0f / (float)(c.g * c.dt * c.dt);
            const float h = (float)c.dt, icm = 1.0f / (float)cm;
            typename Vec4Of<P>::T v4 = s.v[p];
            const float4* prev = aux;  // MODE_FEATURES: previous-correction rows (may be null)
            const float inv3n = fcnt > 0.f ? 1.0f / (3.0f * fcnt) : 0.f;
            float f[32];
            f[0] = (float)d.x * sc; f[1] = (float)d.y * sc; f[2] = (float)d.z * sc;
            f[3] = (float)v4.x * h * sc; f[4] = (float)v4.y * h * sc; f[5] = (float)v4.z * h * sc;
            // the previous step's converged correction (x_end - x0) / s, kept by k_ws_target
            const float4 pc = prev ? prev[p] : make_float4(0.f, 0.f, 0.f, 0.f);
            f[6] = pc.x; f[7] = pc.y; f[8] = pc.z;
            f[9] = fcnt > 0.f ? (fv0 * inv3n - (float)v4.x) * h * sc : 0.f;
            f[10] = fcnt > 0.f ? (fv1 * inv3n - (float)v4.y) * h * sc : 0.f;
            f[11] = fcnt > 0.f ? (fv2 * inv3n - (float)v4.z) * h * sc : 0.f;
            f[12] = (float)rhs.x * icm * sc; f[13] = (float)rhs.y * icm * sc; f[14] = (float)rhs.z * icm * sc;
            f[15] = (float)dx.x * sc; f[16] = (float)dx.y * sc; f[17] = (float)dx.z * sc;
            f[18] = log1pf(fmaxf(0.f, (float)B.h00 * icm));
            f[19] = log1pf(fmaxf(0.f, (float)B.h11 * icm));
            f[20] = log1pf(fmaxf(0.f, (float)B.h22 * icm));
            f[21] = fcnt > 0.f ? fmol / fcnt : 0.f;
            f[22] = log10f((float)m) + 3.0f;
            f[23] = tanhf((float)xi.y * sc * 0.1f);
            f[24] = (GROUND && (fl & VF_GROUND)) ? (float)s.glam[p].x * icm * sc : 0.f;
            f[25] = fcnt * (1.0f / 24.0f);
            f[26] = tanhf((float)y4.y * sc);
#pragma unroll
            for (int j = 27; j < 32; j++) f[j] = 0.f;
            uint32_t w[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                float a = fminf(fmaxf(f[2 * j], -1e4f), 1e4f), b = fminf(fmaxf(f[2 * j + 1], -1e4f), 1e4f);
                if (!(a == a)) a = 0.f;  // a NaN feature becomes 0
                if (!(b == b)) b = 0.f;
                __nv_bfloat162 hb = __floats2bfloat162_rn(a, b);
                w[j] = *reinterpret_cast<uint32_t*>(&hb);
            }
            uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(out) + (size_t)p * 64);
            dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
            dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
            dst[2] = make_uint4(w[8], w[9], w[10], w[11]);
            dst[3] = make_uint4(w[12], w[13], w[14], w[15]);
        } else if constexpr (MODE == MODE_RESIDUAL) {
            double u0 = (double)cm * (double)d.x + (double)B.g0;
            double u1 = (double)cm * (double)d.y + (double)B.g1;
            double u2 = (double)cm * (double)d.z + (double)B.g2;
            r2 = u0 * u0 + u1 * u1 + u2 * u2;
            double mgv = (double)m * (double)c.g;
            mg2 = mgv * mgv;
        } else {
            out[0] = B.g0; out[1] = B.g1; out[2] = B.g2;
            out[3] = B.h00; out[4] = B.h01; out[5] = B.h02;
            out[6] = B.h01; out[7] = B.h11; out[8] = B.h12;
            out[9] = B.h02; out[10] = B.h12; out[11] = B.h22;
        }
    }
    if constexpr (MODE == MODE_RESIDUAL) {
        if (T.ex) {  // per-scene sums
            if (active && lane == 0) {
                if (acc) *acc += r2;
                else atomicAdd(T.ex + T.scene[p], r2);
            }
            return;
        }
        // FP64 reduction: warp, then one atomic per warp
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) {
            r2 += __shfl_xor_sync(0xffffffffu, r2, m);
            mg2 += __shfl_xor_sync(0xffffffffu, mg2, m);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(out, r2);
            atomicAdd(out + 1, mg2);
        }
    }
}

// ranges: when given, block b serves the vertices [x, x + y) of scene z
// (a piece of one scene's part of a color slab) and returns at once when the
// scene is not iterating (solve) or not a residual candidate (residual):
// with per-scene run-to-tolerance most scenes drop out of the later
// iterations, and a block of them then costs one check.  The block's
// residual terms (in-sweep or exact) are summed in registers and reduced
// over the block: one atomic per piece instead of one per vertex on the
// scene's sum.  Otherwise thread groups map to vertices [begin, begin +
// count) (or to list).
// One piece (at most 512 consecutive solved vertices of one scene in one
// color slab) solved by one block; its residual terms are summed over the
// block.  rg = (first vertex, count, scene).
template <typename P, typename RS, typename HT, int LANES, int FORM, bool GROUND, int MODE, bool DYN, bool COH>
__device__ __forceinline__ void solve_piece(const DevState<P>& s, const TetElems<RS>& el, const uint4 rg,
                                            const Consts<P>& c, unsigned long long* counters, double* out,
                                            const SceneTol& T, const float4* __restrict__ aux,
                                            const uint32_t* __restrict__ list) {
    const unsigned lane = threadIdx.x % LANES;
    const uint8_t* gate = MODE == MODE_SOLVE ? T.active : T.cand;
    if (gate && !gate[rg.z]) return;
    double* sum = MODE == MODE_SOLVE ? T.r2 : (MODE == MODE_RESIDUAL ? T.ex : nullptr);
    SceneTol TB = T;  // gated above, for the whole block
    TB.active = nullptr;
    TB.cand = nullptr;
    double acc = 0.0;
    for (unsigned base = 0; base < rg.y; base += blockDim.x / LANES) {
        // this thread group's next vertex is fetched into L2 while this one is
        // solved (its first loads are then not DRAM misses): its whole star
        // form, or the first records
        const unsigned gn = base + blockDim.x / LANES + threadIdx.x / LANES;
        if (gn < rg.y) {
            if constexpr (FORM == FORM_STAR) {
                const uint2 a = el.star[rg.x + gn], b = el.star[rg.x + gn + 1];
                constexpr unsigned SN = 32 / sizeof(StarNb<RS>), ST = 32 / sizeof(StarTet<RS>);
                for (unsigned j = a.x + SN * lane; j < b.x; j += SN * LANES) prefetch_l2(el.nb + j);
                for (unsigned j = a.y + ST * lane; j < b.y; j += ST * LANES) prefetch_l2(el.tet + j);
                for (unsigned j = a.y + 8 * lane; j < b.y; j += 8 * LANES) prefetch_l2(el.loc + j);
            } else {
                const unsigned bn = el.inc_begin[rg.x + gn], en = el.inc_begin[rg.x + gn + 1];
#pragma unroll
                for (unsigned j = 0; j < 4; j++)
                    if (bn + lane + j * LANES < en) prefetch_l2(el.inc + bn + lane + j * LANES);
            }
        }
        tet_vertex<P, RS, HT, LANES, FORM, GROUND, MODE, DYN, COH>(s, el, rg.x, rg.y, base + threadIdx.x / LANES,
                                                                   lane, c, counters, out, TB, aux, list,
                                                                   sum ? &acc : nullptr);
    }
    if (sum) {
        __shared__ double part[32];
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (unsigned w = 0; w < (blockDim.x >> 5); w++) t += part[w];
            atomicAdd(sum + rg.z, t);
        }
    }
}

template <typename P, typename RS, typename HT, int LANES, int FORM, bool GROUND, int MODE, bool DYN>
__global__ void __launch_bounds__(256, (SolveMinBlocks<P, RS, FORM>::value)) k_solve_tet(DevState<P> s, TetElems<RS> el,
                                                   unsigned begin, unsigned count, Consts<P> c,
                                                   unsigned long long* counters, double* out, SceneTol T,
                                                   const float4* __restrict__ aux, const uint32_t* __restrict__ list,
                                                   const uint4* __restrict__ ranges) {
    if (ranges) {
        solve_piece<P, RS, HT, LANES, FORM, GROUND, MODE, DYN, false>(s, el, ranges[blockIdx.x], c, counters, out, T,
                                                                      aux, list);
        return;
    }
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
    tet_vertex<P, RS, HT, LANES, FORM, GROUND, MODE, DYN>(s, el, begin, count, tid / LANES, tid % LANES, c, counters,
                                                          out, T, aux, list);
}

// Polls a grid-barrier wait of k_iterate may take before it gives
// up (avbd_debug_set_wait_limit lowers it so that tests can make it run out).
__device__ uint32_t g_sweep_wait_polls = AVBD_DEFAULT_WAIT_POLLS;

// Dual update of a ground contact at the accelerated position xn
// (CollisionConstraintEnergySolver::updateAfterIteration); true when the
// penalties grew, which they do only in contact: elsewhere k is not stored back.
template <typename R>
AVBD_D bool ground_dual(typename Vec4Of<R>::T& k, typename Vec4Of<R>::T& lam, typename Vec4Of<R>::T cp, uint8_t& gf,
                        V3<R> xn) {
    R Cn = -xn.y, Ct = xn.x - cp.x, Cb = xn.z - cp.y;
    R cc = Cn - R(AVBD_ALPHA) * lam.w;
    R ln = k.x * cc + lam.x;
    R lt = k.y * Ct + lam.y;
    R lb = k.z * Cb + lam.z;
    bool k_grows = ln > R(0);
    bool st = gf & GF_USE_STATIC;
    if (!k_grows && !st) {  // out of contact, sliding coefficient: the cone is a point
        lam.x = R(0);
        lam.y = R(0) * lt;
        lam.z = R(0) * lb;
        gf &= ~GF_UNCLAMPED;
        return false;
    }
    if (ln > R(0)) k.x += R(AVBD_BETA) * fabs(cc);
    lam.x = ln > R(0) ? ln : R(0);
    R mag = sqrt(lt * lt + lb * lb);
    R mx = (st ? cp.z : cp.w) * lam.x;
    if (mag < mx) {
        k_grows = true;
        k.y += R(AVBD_BETA) * fabs(Ct);
        k.z += R(AVBD_BETA) * fabs(Cb);
        lam.y = lt;
        lam.z = lb;
        gf |= GF_UNCLAMPED;
    } else {
        if (st) {
            gf &= ~GF_USE_STATIC;
            mx = cp.w * ln;
        }
        lam.y = lt / (mag + R(1e-8)) * mx;
        lam.z = lb / (mag + R(1e-8)) * mx;
        gf &= ~GF_UNCLAMPED;
    }
    return k_grows;
}

// Chebyshev acceleration of a vertex fused with the ground-contact dual
// update that follows it; a ground energy reads only its own particle, so the
// fusion is exact.
template <typename R>
AVBD_D void chebyshev_dual_vertex(const DevState<R>& s, unsigned p, uint8_t fl, R omega, unsigned it) {
    // o_k = omega (x - o_(k-2)) + o_(k-2); o_k replaces o_(k-2) in its buffer
    typename Vec4Of<R>::T* h = (it & 1u) ? s.xll : s.xl;
    typename Vec4Of<R>::T x4 = s.x[p], ll4 = h[p];
    V3<R> x = xyz(x4), ll = xyz(ll4);
    V3<R> xn = omega * (x - ll) + ll;
    typename Vec4Of<R>::T o = make4<R>(xn, x4.w);
    s.x[p] = o;
    h[p] = o;
    if (fl & VF_GROUND) {
        typename Vec4Of<R>::T k = s.gk[p], lam = s.glam[p], cp = s.gcp[p];
        uint8_t gf = s.gflag[p];
        if (ground_dual<R>(k, lam, cp, gf, xn)) s.gk[p] = k;
        s.glam[p] = lam;
        s.gflag[p] = gf;
    }
}

template <typename R>
__global__ void __launch_bounds__(256) k_chebyshev_dual(DevState<R> s, R omega, unsigned it, SceneTol T) {
    unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n) return;
    uint8_t fl = s.flags[p];
    if (fl & VF_ORIENTED) return;
    if (T.active && !T.active[T.scene[p]]) return;
    if (T.omega) omega = (R)*T.omega;
    if (T.it) it = *T.it;
    chebyshev_dual_vertex<R>(s, p, fl, omega, it);
}

// Barrier over the blocks of an iteration launch.  sync[0] counts arrivals and
// only grows: the barrier numbered b (from 1) opens when it reaches b gridDim.x,
// so one word serves arrival and release.  sync[1] is set by a block whose
// polls ran out; the others see it while they poll, and every block leaves.
AVBD_D bool iterate_barrier(unsigned* sync, unsigned number, int* err) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = number * gridDim.x;
        int good = 1;
        // the block's writes (ordered before by the block barrier) are released
        // with the arrival, the others' acquired with the poll that sees it
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(sync) : "memory");
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(sync) : "memory");
        const unsigned limit = g_sweep_wait_polls;
        for (unsigned polls = 0; (int)(v - target) < 0; polls++) {
            if (polls >= limit || ((polls & 63u) == 63u && *(volatile unsigned*)(sync + 1) != 0)) {
                good = 0;
                break;
            }
            if (polls > 256) __nanosleep(100);
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(sync) : "memory");
        }
        if (!good) {
            atomicExch(sync + 1, 1u);
            atomicCAS(err, 0, (int)AVBD_ERR_BARRIER_TIMEOUT);
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// Threads of an iteration block (one per SM): the prefetching sweeps of the
// star form with a double state take 168 registers (with 128 they spilled and
// a batch of 24 scenes ran 10.3 instead of 7.3 ms a pass), the others 128.
// FP32 records at 2 lanes, which large colors take, stream better at twice the
// warps, 64 registers and some 100 bytes of spill (to 1e-4 241,611 vertices a
// color 57.9 with 512 threads and 51.9 ms a step, 481,124 106.9 and 91.8); MIXED
// ones did not (24 scenes 11.5 ms, 15.6 with 768 threads).
template <typename P, int FORM, int LANES = 8>
struct IterThreads {
    static constexpr int value = FORM == FORM_STAR && sizeof(P) == 8 && LANES > 2 ? 384
                                 : FORM != FORM_STAR && sizeof(P) == 4 && LANES == 2 ? 1024 : 512;
};

// A piece of 32 / LANES vertices of the star form whose constant data are on
// their way into registers: this thread's entries of the first rounds (16
// neighbours and 24 tets a vertex; the rest is read when its turn comes).
template <typename RS, int LANES>
struct StarPiece {
    static constexpr int UN = 16 / LANES, UT = 24 / LANES;
    uint4 h;  // TetElems::piece
    StarNb<RS> nb[UN];
    StarTet<RS> tet[UT];
    uint32_t loc[UT];

    AVBD_D void lists(const TetElems<RS>& el, unsigned wl) {
#pragma unroll
        for (int u = 0; u < UN; u++)
            if (u < (int)h.y) nb[u] = ld_once(el.pnb + h.x + u * 32 + wl);
#pragma unroll
        for (int u = 0; u < UT; u++)
            if (u < (int)h.w) {
                tet[u] = ld_once(el.ptet + h.z + u * 32 + wl);
                loc[u] = ld_once(el.ploc + h.z + u * 32 + wl);
            }
    }
};

// Staging rows of k_iterate: whole rounds of LANES neighbours.
AVBD_HD unsigned star_rows(unsigned max_nb, unsigned lanes) { return (max_nb + lanes - 1) / lanes * lanes; }

// Arguments of an iteration launch.
struct IterArgs {
    const uint4* slabs;       // per color: first internal vertex, solved positional vertices, first piece
    unsigned ncolors;
    const double* omega;      // Chebyshev weights by iteration
    unsigned it0, n;          // first iteration, iterations at most
    bool sweep_only;          // the solves alone (lane choice): histories and multipliers untouched
    unsigned* sync;           // barrier, zeroed before
    // run to tolerance
    unsigned max_it;          // iteration cap of the step
    uint32_t* it_dev;         // loop of a graph: first iteration from device memory, advanced at the end
    double tol, g2;
    const double* m2;
    uint8_t *active, *cand;
    uint32_t* iters;
    double *r2, *ex, *rin;    // r2: 3 buffers of S by iteration, ex: 2 by residual pass (k_iterate)
    unsigned S;
    unsigned long long* scene_iterations;
    unsigned long long* maxr;
    int* n_active;
    cudaGraphConditionalHandle loop;  // continue condition of the graph's loop (has_loop)
    bool has_loop;
    unsigned long long* launches;
};

AVBD_D double scene_R(double r2, double mg2) { return mg2 > 0 ? sqrt(r2) / sqrt(mg2) : sqrt(r2); }

AVBD_D unsigned long long ord_enc64(double d) {
    unsigned long long u = (unsigned long long)__double_as_longlong(d);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// Residual terms of a warp's consecutive pieces, one atomic per scene run.
struct SceneSum {
    double* sums;
    unsigned run = 0xFFFFFFFFu;
    double racc = 0.0;
    AVBD_D SceneSum(double* s) : sums(s) {}
    AVBD_D void flush() {
        double t = racc;
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) t += __shfl_xor_sync(0xffffffffu, t, m);
        if ((threadIdx.x & 31u) == 0 && run != 0xFFFFFFFFu) atomicAdd(sums + run, t);
        run = 0xFFFFFFFFu;
        racc = 0.0;
    }
    AVBD_D void add(unsigned scene, double term) {
        const unsigned sc0 = __shfl_sync(0xffffffffu, scene, 0);
        if (__all_sync(0xffffffffu, scene == sc0)) {
            if (sc0 != run) {
                flush();
                run = sc0;
            }
            racc += term;
        } else if (term != 0.0) {
            atomicAdd(sums + scene, term);
        }
    }
};

// Scenes as bits in shared memory: every block keeps its own copy of which
// scenes iterate and which are candidates, computed from the same sums.
struct SceneBits {
    uint32_t* w;
    AVBD_D bool get(unsigned s) const { return w[s >> 5] >> (s & 31u) & 1u; }
};

// The solved vertices [begin, begin + count) of a color in MODE, a warp taking
// 32 / LANES consecutive ones at a time (see k_iterate).  TOL: vertices of
// scenes outside the gate are skipped; the residual terms go to the scenes' sums.
template <typename P, typename RS, typename HT, int LANES, int FORM, bool GROUND, bool TOL, int MODE>
AVBD_D void color_phase(const DevState<P>& s, const TetElems<RS>& el, const Consts<P>& c,
                        unsigned long long* counters, const uint32_t* scene, unsigned begin, unsigned count,
                        SceneBits gate, double* sums, bool spread) {
    constexpr int THREADS = IterThreads<P, FORM, LANES>::value;
    constexpr unsigned WARPS = THREADS / 32, V = 32 / LANES;
    const unsigned warp = threadIdx.x >> 5, wl = threadIdx.x & 31u, lane = wl % LANES;
    const unsigned B = gridDim.x, b = blockIdx.x;
    const unsigned nch = (count + V - 1) / V;
    const unsigned per = (nch + B - 1) / B;
    unsigned k = spread ? b * WARPS + warp : b * per + warp;
    const unsigned end = spread ? nch : min(nch, (b + 1) * per);
    const unsigned step = spread ? B * WARPS : WARPS;
    SceneSum sum(sums);
    SceneTol TB;
    if constexpr (TOL) {
        TB.r2 = MODE == MODE_SOLVE ? sums : nullptr;
        TB.ex = MODE == MODE_RESIDUAL ? sums : nullptr;
        TB.scene = scene;
    }
    for (; k < end; k += step) {
        unsigned gi = k * V + wl / LANES;
        unsigned sc = 0;
        if constexpr (TOL) {
            sc = scene[begin + min(gi, count - 1)];
            if (!gate.get(sc)) gi = count;
            if (!__any_sync(0xffffffffu, gi < count)) continue;
        }
        double acc = 0.0;
        tet_vertex<P, RS, HT, LANES, FORM, GROUND, MODE, false, true, THREADS>(
            s, el, begin, count, gi, lane, c, counters, nullptr, TB, nullptr, nullptr, TOL ? &acc : nullptr);
        if constexpr (TOL) {
            __syncwarp();
            sum.add(sc, acc);
        }
    }
    if constexpr (TOL) sum.flush();
}

// The exact residual of the candidate scenes: rare, and kept out of line so
// that it takes no registers from the sweeps.
template <typename P, typename RS, typename HT, int LANES, int FORM, bool GROUND>
__device__ __noinline__ void residual_phase(const DevState<P>& s, const TetElems<RS>& el, const Consts<P>& c,
                                            const uint32_t* scene, const IterArgs& A, SceneBits cand, double* ex) {
    for (unsigned col = 0; col < A.ncolors; col++) {
        const uint4 sl = A.slabs[col];
        if (sl.y)
            color_phase<P, RS, HT, LANES, FORM, GROUND, true, MODE_RESIDUAL>(s, el, c, nullptr, scene, sl.x, sl.y,
                                                                             cand, ex, true);
    }
}

// After a sweep: an iterating scene whose in-sweep residual is at the
// tolerance becomes a candidate.  Returns the number of candidates (uniform
// over the block).
__device__ __noinline__ unsigned iterate_candidates(const IterArgs& A, SceneBits on, SceneBits cand, const double* r2,
                                                    unsigned* red) {
    for (unsigned i = threadIdx.x; i < (A.S + 31) / 32; i += blockDim.x) cand.w[i] = 0;
    if (threadIdx.x == 0) *red = 0;
    __syncthreads();
    const double t2 = A.tol * A.tol * (1 + 1e-9);  // a cheap bound first, then the exact comparison
    unsigned n = 0;
    for (unsigned q = threadIdx.x; q < A.S; q += blockDim.x)
        if (on.get(q)) {
            const double r = __ldcg(r2 + q), mg2 = A.m2[q] * A.g2;  // 0 without gravity: the residual is absolute
            if ((r <= t2 * mg2 || !(mg2 > 0)) && scene_R(r, mg2) <= A.tol) {
                atomicOr(cand.w + (q >> 5), 1u << (q & 31u));
                n++;
            }
        }
    if (n) atomicAdd(red, n);
    __syncthreads();
    const unsigned total = *red;
    __syncthreads();  // red may be reused
    return total;
}

// Stop decision: candidates whose exact residual is at the tolerance stop; at
// the iteration cap every scene does.  The recording block also stores the
// scenes' iteration counts, the step's largest final residual (maxr[0]: the
// exact one where it was evaluated in the stopping iteration, else the
// in-sweep one of a capped scene) and the number of capped scenes (maxr[1]).
// Returns the number of scenes that stopped.
__device__ __noinline__ unsigned iterate_stop(const IterArgs& A, SceneBits on, SceneBits cand, const double* r2,
                                              const double* ex, unsigned iters, bool record, unsigned* red) {
    if (threadIdx.x == 0) *red = 0;
    __syncthreads();
    const bool cap = iters >= A.max_it;
    unsigned n = 0;
    for (unsigned q = threadIdx.x; q < A.S; q += blockDim.x) {
        if (!on.get(q)) continue;
        const bool cd = cand.get(q);
        if (!cd && !cap) continue;
        const double R = scene_R(__ldcg((cd ? ex : r2) + q), A.m2[q] * A.g2);
        const bool met = cd && R <= A.tol;
        if (!met && !cap) continue;
        n++;
        atomicAnd(on.w + (q >> 5), ~(1u << (q & 31u)));
        if (record) {
            A.iters[q] = iters;
            atomicMax(A.maxr, ord_enc64(R));
            if (!met) atomicAdd(A.maxr + 1, 1ull);
        }
    }
    if (n) atomicAdd(red, n);
    __syncthreads();
    const unsigned total = *red;
    __syncthreads();
    return total;
}

// 32-byte accesses of a vertex record of four doubles (float4 is one already).
// Loads are coherent: other blocks of the launch write the positions.
AVBD_D float4 ld_vec(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
AVBD_D double4a ld_vec(const double4a* p) {
    double4a v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
AVBD_D void st_vec(float4* p, float4 v) { *p = v; }
AVBD_D void st_vec(double4a* p, double4a v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v.x), "d"(v.y), "d"(v.z), "d"(v.w) : "memory");
}

// What follows the accumulated block of a vertex in k_iterate: the 3x3 solve,
// the solved position for the later colors, the accelerated one and the
// history for the next iteration.  Returns the accelerated position.
template <typename P, typename HT>
AVBD_D V3<P> block_rhs(const Block3<P, HT>& B, V3<P> xi, typename Vec4Of<P>::T y4, P inv_dt2) {
    const P cm = y4.w * inv_dt2;
    const V3<P> d = xi - xyz(y4);
    return mk3<P>(-cm * d.x - B.g0, -cm * d.y - B.g1, -cm * d.z - B.g2);
}
template <typename P>
AVBD_D double sum_sq(V3<P> v) {
    return (double)v.x * (double)v.x + (double)v.y * (double)v.y + (double)v.z * (double)v.z;
}
template <typename P, typename HT>
AVBD_D V3<P> finish_vertex(const DevState<P>& s, const Consts<P>& c, const IterArgs& A, unsigned long long* counters,
                           const Block3<P, HT>& B, V3<P> rhs, V3<P> xi, unsigned p, P mass, V3<P> h, P om,
                           typename Vec4Of<P>::T* hist) {
    const P cm = mass * c.inv_dt2;
    Sym3<P> M{cm + (P)B.h00, cm + (P)B.h11, cm + (P)B.h22, (P)B.h01, (P)B.h02, (P)B.h12};
    V3<P> dx;
    if (!solve_sym3<P>(M, rhs, c.kappa_max, dx)) dx = solve_block_d(M, rhs, counters);
    const V3<P> xs = xi + dx;
    st_vec(s.x + s.n + p, make4<P>(xs, P(0)));
    const V3<P> xa = A.sweep_only ? xs : om * (xs - h) + h;
    const typename Vec4Of<P>::T o = make4<P>(xa, P(0));
    st_vec(s.x + p, o);
    if (!A.sweep_only) st_vec(hist + p, o);
    return xa;
}
// The ground contact's duals at the accelerated position; what does not change
// (most vertices are out of contact) is not stored back.
template <typename P>
AVBD_D void finish_ground(const DevState<P>& s, unsigned p, typename Vec4Of<P>::T k, typename Vec4Of<P>::T lam,
                          typename Vec4Of<P>::T cp, uint8_t gf, V3<P> xa) {
    const uint8_t g0 = gf;
    const V3<P> l0 = xyz(lam);
    if (ground_dual<P>(k, lam, cp, gf, xa)) st_vec(s.gk + p, k);
    if (l0.x != lam.x || l0.y != lam.y || l0.z != lam.z) st_vec(s.glam + p, lam);
    if (gf != g0) s.gflag[p] = gf;
}

// The iterations of a step in one cooperative launch of a block per SM, with a
// grid barrier between colors (about 1 us, against about 3 us for a launch of
// a graph).  Small scenes are bounded by these phases, not by their bytes: what
// follows a barrier is a chain of round trips to L2 and of FP64 latencies.
//
// Star form: the Chebyshev acceleration and the ground duals need only the
// vertex's own solved position, so they follow its solve instead of taking a
// pass and a barrier of their own: the solved position goes to the second half
// of x, where the later colors of this iteration read it (tagged ids, StarNb),
// the accelerated one to x itself, for the next iteration.  A warp's pieces
// (32 / LANES consecutive vertices) run as one sequence over the colors: the next piece's header is loaded while the current one
// gathers, its lists while the current one reduces and solves -- also across
// the barrier, since they are constant -- so a phase is one round trip for the
// positions and the arithmetic.  Measured: a barrier with the release and the
// first read behind it 1.9 us, a color of an 8^3 cube 2.9 us (4.6 with the
// loads of the lists behind the barrier, 3.7 as a launch of a graph).
// Records: every color is a pass of tet_vertex and the acceleration another.  So
// does the star form at 2 lanes, which only AVBD_LANES=2 takes: it solves as
// k_solve_tet does, operation for operation, so that the two can be compared.
//
// While every scene iterates, the blocks own contiguous parts of a color
// (neighbouring vertices share their neighbours in L1); once scenes have
// stopped the pieces are dealt round robin, which spreads the remaining scenes
// over the SMs.  TOL: scenes run to their residual tolerance.  Every block
// evaluates the decisions itself from the scenes' sums (3 buffers by
// iteration, so that none is cleared while another block reads it); only an
// iteration with candidates pays for the exact residual and a barrier.
template <typename P, typename RS, typename HT, int LANES, int FORM, bool GROUND, bool TOL>
__global__ void __launch_bounds__((IterThreads<P, FORM, LANES>::value), 1)
    k_iterate(const __grid_constant__ DevState<P> s, const __grid_constant__ TetElems<RS> el,
              const __grid_constant__ Consts<P> c, unsigned long long* counters, const uint32_t* scene,
              const __grid_constant__ IterArgs A) {
    using V4 = typename Vec4Of<P>::T;
    constexpr int THREADS = IterThreads<P, FORM, LANES>::value;
    constexpr unsigned WARPS = THREADS / 32, V = 32 / LANES;
    constexpr bool PIPE = FORM == FORM_STAR && LANES > 2;  // accelerates as it solves
    constexpr unsigned ST = StarStage<P, LANES, THREADS>::STRIDE;
    using Piece = StarPiece<RS, PIPE ? LANES : 4>;
    __shared__ unsigned red;
    __shared__ uint4 slabs[256];  // A.slabs: a load from global memory at each phase would sit on its chain
    extern __shared__ __align__(16) unsigned char stage[];
    for (unsigned q = threadIdx.x; q < A.ncolors; q += blockDim.x) slabs[q] = A.slabs[q];
    __syncthreads();
    const unsigned warp = threadIdx.x >> 5, wl = threadIdx.x & 31u, lane = wl % LANES;
    const unsigned B = gridDim.x, b = blockIdx.x;
    const unsigned K = PIPE ? star_rows(el.max_nb, LANES) : el.max_nb;
    P* const es = reinterpret_cast<P*>(stage) + threadIdx.x / LANES;
    unsigned bar = 0;
    const unsigned first = TOL && A.it_dev ? *A.it_dev : A.it0;
    unsigned last = first + A.n;
    if (TOL && last > A.max_it) last = A.max_it;
    unsigned it = first, na = 0, exn = 0;
    unsigned done_it = 0;  // scene-iterations of this launch
    SceneBits on{nullptr}, cand{nullptr};
    if constexpr (TOL) {
        // a block that leaves at a barrier ends the graph's loop: the condition
        // is only set again once the launch has run to its end
        if (A.has_loop && b == B - 1 && threadIdx.x == 0) cudaGraphSetConditional(A.loop, 0u);
        on.w = reinterpret_cast<uint32_t*>(stage + (FORM == FORM_STAR ? 3 * K * ST * sizeof(P) : 0));
        cand.w = on.w + (A.S + 31) / 32;
        for (unsigned q0 = warp * 32; q0 < A.S; q0 += THREADS) {
            const unsigned m = __ballot_sync(0xffffffffu, q0 + wl < A.S && A.active[min(q0 + wl, A.S - 1)]);
            if (wl == 0) on.w[q0 >> 5] = m;
        }
        na = (unsigned)*A.n_active;
        // the first residual pass adds to buffer 0 (a barrier away)
        if (b == B - 1)
            for (unsigned q = threadIdx.x; q < A.S; q += THREADS) A.ex[q] = 0;
        __syncthreads();
    }

    Piece cur;
    // `cur` is piece ck of phase cphase; this thread's vertex of it, solved when clive
    unsigned ck = 0, cend = 0, cstep = 0, cbegin = 0, ccount = 1, cpiece = 0, cphase = 0, cp = 0;
    bool clive = false;
    auto next_color = [&](unsigned col) {  // the next color with vertices, cyclic
        do col = col + 1 < A.ncolors ? col + 1 : 0;
        while (slabs[col].y == 0);
        return col;
    };
    auto load_header = [&](bool spread) {  // of piece ck; stopped scenes' pieces are passed over
        for (; ck < cend; ck += cstep) {
            const unsigned gi = ck * V + wl / LANES;
            clive = gi < ccount;
            cp = cbegin + min(gi, ccount - 1);
            if constexpr (TOL)
                if (spread) {
                    clive = clive && on.get(scene[cp]);
                    if (!__any_sync(0xffffffffu, clive)) continue;
                }
            cur.h = el.piece[cpiece + ck];
            return;
        }
    };
    auto start_color = [&](unsigned col, bool spread, unsigned phase) {
        const uint4 sl = slabs[col];
        const unsigned nch = (sl.y + V - 1) / V, per = (nch + B - 1) / B;
        cbegin = sl.x;
        ccount = sl.y;
        cpiece = sl.z;
        cphase = phase;
        ck = spread ? b * WARPS + warp : b * per + warp;
        cend = spread ? nch : min(nch, (b + 1) * per);
        cstep = spread ? B * WARPS : WARPS;
        load_header(spread);
    };

    bool spread = TOL && na < A.S;
    unsigned phase = 0;
    const unsigned color0 = next_color(A.ncolors - 1);
    if constexpr (PIPE) {
        start_color(color0, spread, phase);
        if (ck < cend) cur.lists(el, wl);
    }
    for (; it < last && (!TOL || na > 0); it++) {
        double* const r2 = TOL ? A.r2 + (size_t)(it % 3u) * A.S : nullptr;
        if constexpr (TOL) done_it += na;
        const P om = A.sweep_only ? P(1) : (P)A.omega[it];
        if constexpr (PIPE) {
            V4* const hist = (it & 1u) ? s.xll : s.xl;
            SceneSum sum(r2);
            for (unsigned col = 0; col < A.ncolors; col++) {
                if (slabs[col].y == 0) continue;
                while (cphase == phase && ck < cend) {
                    const unsigned p = cp;
                    const bool live = clive;
                    const uint4 h = cur.h;
                    Block3<P, HT> Bk;
                    // positions, then what lanes 0 (inertia, history) and 1 (ground contact) add
                    const V3<P> xi = xyz(ld_vec(s.x + p));
                    V3<P> xo[Piece::UN];
#pragma unroll
                    for (int u = 0; u < Piece::UN; u++)
                        if (u < (int)h.y) xo[u] = xyz(ld_vec(s.x + cur.nb[u].idx));
                    V4 r0 = make4<P>(mk3<P>(0, 0, 0), P(0)), r1 = r0, r2v = r0;  // y, history | gcp, k, lambda
                    HT hd = 0;
                    uint8_t fl = 0, gf = 0;
                    if (live && lane == 0) {
                        r0 = ld_vec(s.y + p);
                        r1 = ld_vec(hist + p);
                        hd = (HT)el.hd[p];
                    }
                    if (GROUND && live && lane == 1) {
                        fl = s.flags[p];
                        r0 = ld_vec(s.gcp + p);
                        r1 = ld_vec(s.gk + p);
                        r2v = ld_vec(s.glam + p);
                        gf = s.gflag[p];
                    }
                    RS w[Piece::UN];
#pragma unroll
                    for (int u = 0; u < Piece::UN; u++) w[u] = cur.nb[u].w;
                    // the next piece: of this color, else the first of the next
                    ck += cstep;
                    load_header(spread);
                    if (ck >= cend) start_color(next_color(col), spread, phase + 1);
#pragma unroll
                    for (int u = 0; u < Piece::UN; u++)
                        if (u < (int)h.y)
                            star_edge<P, RS, HT, ST>(w[u], xo[u] - xi, es + (lane + u * LANES) * ST, K, Bk);
                    for (unsigned u = Piece::UN; u < h.y; u++) {
                        const StarNb<RS> q = ld_once(el.pnb + h.x + u * 32 + wl);
                        star_edge<P, RS, HT, ST>(q.w, xyz(ld_vec(s.x + q.idx)) - xi, es + (lane + u * LANES) * ST, K, Bk);
                    }
                    __syncwarp();
#pragma unroll
                    for (int u = 0; u < Piece::UT; u++)
                        if (u < (int)h.w) star_tet<P, RS, HT, ST>(cur.tet[u], cur.loc[u], es, K, Bk);
                    for (unsigned u = Piece::UT; u < h.w; u++)
                        star_tet<P, RS, HT, ST>(ld_once(el.ptet + h.z + u * 32 + wl),
                                                ld_once(el.ploc + h.z + u * 32 + wl), es, K, Bk);
                    __syncwarp();  // the slot is refilled for the next piece
                    if (ck < cend) cur.lists(el, wl);
                    if (GROUND && (fl & VF_GROUND)) accumulate_ground<P, HT>(r1, r2v, r0, gf, xi, Bk);
                    Bk.h00 += hd;
                    Bk.h11 += hd;
                    Bk.h22 += hd;
                    reduce_block<LANES>(Bk);
                    double acc = 0.0;
                    V3<P> xa = xi;
                    if (live && lane == 0) {
                        const V3<P> rhs = block_rhs(Bk, xi, r0, c.inv_dt2);
                        if (TOL) acc = sum_sq(rhs);
                        xa = finish_vertex<P, HT>(s, c, A, counters, Bk, rhs, xi, p, r0.w, xyz(r1), om, hist);
                    }
                    if constexpr (GROUND) {
                        xa.x = __shfl_sync(0xffffffffu, xa.x, wl & ~(LANES - 1));
                        xa.y = __shfl_sync(0xffffffffu, xa.y, wl & ~(LANES - 1));
                        xa.z = __shfl_sync(0xffffffffu, xa.z, wl & ~(LANES - 1));
                        if ((fl & VF_GROUND) && !A.sweep_only) finish_ground<P>(s, p, r1, r2v, r0, gf, xa);
                    }
                    const unsigned sc = TOL ? scene[p] : 0u;
                    if constexpr (TOL) {
                        __syncwarp();
                        sum.add(sc, acc);
                    }
                }
                if constexpr (TOL) sum.flush();
                if (cphase == phase) {  // a warp without a piece in this color
                    start_color(next_color(col), spread, phase + 1);
                    if (ck < cend) cur.lists(el, wl);
                }
                phase++;
                if (!iterate_barrier(A.sync, ++bar, s.err)) return;
            }
        } else {
            for (unsigned col = 0; col < A.ncolors; col++) {
                const uint4 sl = slabs[col];
                if (sl.y == 0) continue;
                color_phase<P, RS, HT, LANES, FORM, GROUND, TOL, MODE_SOLVE>(s, el, c, counters, scene, sl.x, sl.y, on,
                                                                             r2, spread);
                if (!iterate_barrier(A.sync, ++bar, s.err)) return;
            }
            if (A.sweep_only) continue;
            for (unsigned p = b * THREADS + threadIdx.x; p < s.n; p += B * THREADS) {
                if (TOL && !on.get(scene[p])) continue;
                chebyshev_dual_vertex<P>(s, p, GROUND ? s.flags[p] : (uint8_t)0, om, it);
            }
            if (!iterate_barrier(A.sync, ++bar, s.err)) return;
        }
        if constexpr (TOL) {
            // the buffer of the iteration after the next: last read a barrier ago
            if (b == B - 1)
                for (unsigned q = threadIdx.x; q < A.S; q += THREADS) A.r2[(size_t)((it + 2) % 3u) * A.S + q] = 0;
            const unsigned nc = iterate_candidates(A, on, cand, r2, &red);
            if (nc == 0 && it + 1 < A.max_it) continue;
            double* const ex = A.ex + (size_t)(exn & 1u) * A.S;
            if (nc) {
                if (b == B - 1)  // the other buffer, last read before the sweep
                    for (unsigned q = threadIdx.x; q < A.S; q += THREADS) A.ex[(size_t)(~exn & 1u) * A.S + q] = 0;
                residual_phase<P, RS, HT, LANES, FORM, GROUND>(s, el, c, scene, A, cand, ex);
                if (!iterate_barrier(A.sync, ++bar, s.err)) return;
                exn++;
            }
            na -= iterate_stop(A, on, cand, r2, ex, it + 1, b == B - 1, &red);
            if (na > 0 && na < A.S) {  // scenes have stopped: other pieces than those on their way
                spread = true;
                if constexpr (PIPE) {
                    start_color(color0, spread, phase);
                    if (ck < cend) cur.lists(el, wl);
                }
            }
        }
    }
    if (TOL && b == B - 1) {
        for (unsigned q = threadIdx.x; q < A.S; q += THREADS) {
            const bool live = on.get(q);
            A.active[q] = live;
            if (live) A.iters[q] = it;
        }
        if (threadIdx.x == 0) {
            *A.n_active = (int)na;
            *A.scene_iterations += done_it;
            if (A.it_dev) *A.it_dev = it;
            if (A.has_loop) {
                *A.launches += 1;
                cudaGraphSetConditional(A.loop, na > 0 && it < A.max_it ? 1u : 0u);
            }
        }
    }
}

template <typename R>
__global__ void __launch_bounds__(256) k_velocity(DevState<R> s, R inv_dt) {
    unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n) return;
    if (s.flags[p] & VF_ORIENTED) return;
    typename Vec4Of<R>::T x4 = s.x[p], xp4 = s.xp[p];
    s.vp[p] = s.v[p];
    s.v[p] = make4<R>(inv_dt * (xyz(x4) - xyz(xp4)), R(0));
    s.xp[p] = x4;
    if (!isfinite(x4.x + x4.y + x4.z)) atomicExch(s.err, (int)AVBD_ERR_NAN);
}

// Host FP64 (external order) -> device state.  mode 0: positions only,
// mode 1: positions and every derived position array (ParticlePool::addParticle
// reset), mode 2: velocities (src) and previous velocities (src + 3n),
// mode 3: velocities only.
template <typename R>
__global__ void k_load(DevState<R> s, const double* src, const uint32_t* inv_map, unsigned first, unsigned n,
                       int mode) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned p = inv_map[first + i];
    V3<R> v = mk3<R>((R)src[3 * i], (R)src[3 * i + 1], (R)src[3 * i + 2]);
    if (mode == 2) {
        V3<R> w = mk3<R>((R)src[3 * (n + i)], (R)src[3 * (n + i) + 1], (R)src[3 * (n + i) + 2]);
        s.v[p] = make4<R>(v, R(0));
        s.vp[p] = make4<R>(w, R(0));
        return;
    }
    if (mode == 3) {
        s.v[p] = make4<R>(v, R(0));
        return;
    }
    typename Vec4Of<R>::T o = make4<R>(v, R(0));
    if (mode == 4) {  // a caller's initial guess of the step: solved positional vertices only
        if (s.flags[p] & (VF_FIXED | VF_ORIENTED)) return;
        s.x[p] = o;
        s.xl[p] = o;
        s.xll[p] = o;
        return;
    }
    s.x[p] = o;
    if (mode == 1) {
        typename Vec4Of<R>::T y4 = s.y[p];
        s.y[p] = make4<R>(v, y4.w);
        s.xp[p] = o;
        s.xl[p] = o;
        s.xll[p] = o;
    }
}

// Device state -> host FP64 (external order).  which: 0 x, 1 v, 2 xp.
template <typename R>
__global__ void k_store(DevState<R> s, int which, double* dst, const uint32_t* inv_map, unsigned first, unsigned n) {
    unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned p = inv_map[first + i];
    typename Vec4Of<R>::T a = which == 0 ? s.x[p] : which == 1 ? s.v[p] : s.xp[p];
    dst[3 * i] = (double)a.x;
    dst[3 * i + 1] = (double)a.y;
    dst[3 * i + 2] = (double)a.z;
}

// ---------------------------------------------------------------- host
template <typename R>
void launch_begin_step(avbd_ctx* c, DevState<R>& s, const StepConsts& k, cudaStream_t st) {
    k_begin_step<R><<<nblocks(s.n, 256), 256, 0, st>>>(s, mkc<R>(k));
    count_launch(c);
}

template <typename R>
void launch_tet_eprev(avbd_ctx* c, DevState<R>& s, const StepConsts& k, cudaStream_t st) {
    (void)k;
    if (s.ntets == 0) return;
    k_tet_eprev<R><<<nblocks(s.ntets, 256), 256, 0, st>>>(s);
    count_launch(c);
}

// Dynamic shared memory a kernel's neighbour staging may take: what a block can
// have (227 KB) less the static part of these kernels (under 8 KB).
constexpr unsigned STAGE_SMEM_MAX = (227 - 8) * 1024;
// Above 48 KB with the static part a kernel has to opt in.  The limit belongs to
// the kernel, which all contexts and host threads of the process share, so it
// is only ever set to this one value: set to a context's own size, a smaller
// context could lower it between a larger one's setting and its launch.
template <typename K>
static bool stage_smem(K kern, unsigned bytes) {
    return bytes <= 40 * 1024 ||
           (bytes <= STAGE_SMEM_MAX &&
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STAGE_SMEM_MAX) == cudaSuccess);
}

template <typename P, typename RS, typename HT, int LANES, int FORM, int MODE, bool DYN>
static void solve_dispatch_form(avbd_ctx* c, DevState<P>& s, const TetElems<RS>& el, const StepConsts& k,
                                unsigned begin, unsigned count, cudaStream_t st, double* out, const SceneTol& T,
                                const uint32_t* list, const uint4* ranges, unsigned nranges) {
    const unsigned blocks = ranges ? nranges : nblocks(count * LANES, 256);
    if (blocks == 0) return;
    const unsigned smem = FORM == FORM_STAR ? StarStage<P, LANES>::bytes(el.max_nb) : 0;
    auto kern = c->ground.empty() ? k_solve_tet<P, RS, HT, LANES, FORM, false, MODE, DYN>
                                  : k_solve_tet<P, RS, HT, LANES, FORM, true, MODE, DYN>;
    // a kernel that cannot have its shared memory fails at the launch, which the step checks
    stage_smem(kern, smem);
    kern<<<blocks, 256, smem, st>>>(s, el, begin, count, mkc<P>(k), c->d_counters, out, T,
                                    reinterpret_cast<const float4*>(c->ws_prev_arg), list, ranges);
    count_launch(c);
}

template <typename P, typename RS, typename HT, int LANES, int MODE, bool DYN = false>
static void solve_dispatch(avbd_ctx* c, DevState<P>& s, const TetElems<RS>& el, const StepConsts& k, unsigned begin,
                           unsigned count, cudaStream_t st, double* out, const SceneTol& T, const uint32_t* list,
                           const uint4* ranges = nullptr, unsigned nranges = 0) {
    if (el.star)
        solve_dispatch_form<P, RS, HT, LANES, FORM_STAR, MODE, DYN>(c, s, el, k, begin, count, st, out, T, list, ranges, nranges);
    else if (c->damping)
        solve_dispatch_form<P, RS, HT, LANES, FORM_DAMP, MODE, DYN>(c, s, el, k, begin, count, st, out, T, list, ranges, nranges);
    else
        solve_dispatch_form<P, RS, HT, LANES, FORM_REC, MODE, DYN>(c, s, el, k, begin, count, st, out, T, list, ranges, nranges);
}

// The solve, residual and features passes run with the context's lane count
// (the residual pass spans every vertex every iteration, so its thread count
// matters even when few scenes are candidates); the one-vertex debug pass
// uses 8.
template <typename P, typename RS, typename HT, int MODE>
static void solve_lanes_t(avbd_ctx* c, DevState<P>& s, const TetElems<RS>& el, const StepConsts& k, unsigned begin,
                          unsigned count, cudaStream_t st, double* out, const SceneTol& T, const uint32_t* list,
                          const uint4* ranges = nullptr, unsigned nranges = 0) {
    if constexpr (MODE == MODE_RESIDUAL) {  // tolerance residual: the sweeps' per-scene pieces, all colors
        if (!list && T.cand && T.ex && c->d_solve_ranges) {
            ranges = c->d_solve_ranges;
            nranges = c->solve_range_off.back();
        }
    }
    if constexpr (MODE == MODE_DEBUG) {
        if (c->dyn) solve_dispatch<P, RS, HT, 8, MODE, true>(c, s, el, k, begin, count, st, out, T, list);
        else solve_dispatch<P, RS, HT, 8, MODE>(c, s, el, k, begin, count, st, out, T, list);
    } else if (list) {
        if constexpr (MODE == MODE_SOLVE || MODE == MODE_RESIDUAL)
            solve_dispatch<P, RS, HT, 8, MODE, true>(c, s, el, k, begin, count, st, out, T, list);
    } else {
        switch (c->lanes) {
            case 2: solve_dispatch<P, RS, HT, 2, MODE>(c, s, el, k, begin, count, st, out, T, list, ranges, nranges); break;
            case 4: solve_dispatch<P, RS, HT, 4, MODE>(c, s, el, k, begin, count, st, out, T, list, ranges, nranges); break;
            case 16: solve_dispatch<P, RS, HT, 16, MODE>(c, s, el, k, begin, count, st, out, T, list, ranges, nranges); break;
            default: solve_dispatch<P, RS, HT, 8, MODE>(c, s, el, k, begin, count, st, out, T, list, ranges, nranges); break;
        }
    }
}

// FP32: everything in float.  FP64: everything in double.  Mixed: double
// state and gradient, float records and Hessian.
template <int MODE>
static void solve_lanes(avbd_ctx* c, DevState<float>& s, const StepConsts& k, unsigned begin, unsigned count,
                        cudaStream_t st, double* out, const SceneTol& T, const uint32_t* list = nullptr,
                        const uint4* ranges = nullptr, unsigned nranges = 0) {
    solve_lanes_t<float, float, float, MODE>(c, s, s.el, k, begin, count, st, out, T, list, ranges, nranges);
}
template <int MODE>
static void solve_lanes(avbd_ctx* c, DevState<double>& s, const StepConsts& k, unsigned begin, unsigned count,
                        cudaStream_t st, double* out, const SceneTol& T, const uint32_t* list = nullptr,
                        const uint4* ranges = nullptr, unsigned nranges = 0) {
    if (c->solver.precision == AVBD_PRECISION_MIXED)
        solve_lanes_t<double, float, float, MODE>(c, s, s.el32, k, begin, count, st, out, T, list, ranges, nranges);
    else
        solve_lanes_t<double, double, double, MODE>(c, s, s.el, k, begin, count, st, out, T, list, ranges, nranges);
}

int solve_set_wait_limit(unsigned polls) {
    cudaError_t e = cudaMemcpyToSymbol(g_sweep_wait_polls, &polls, sizeof(polls));
    return e == cudaSuccess ? AVBD_OK : set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
}

template <typename R>
void launch_solve_color(avbd_ctx* c, DevState<R>& s, const StepConsts& k, unsigned begin, unsigned count,
                        cudaStream_t st, const SceneTol& T, const uint32_t* list, const uint4* ranges,
                        unsigned nranges) {
    solve_lanes<MODE_SOLVE>(c, s, k, begin, count, st, nullptr, T, list, ranges, nranges);
}

template <typename R>
void launch_chebyshev_dual(avbd_ctx* c, DevState<R>& s, const StepConsts& k, double omega, unsigned it,
                           cudaStream_t st, const SceneTol& T) {
    (void)k;
    if (s.no == s.n) return;  // every particle oriented: k_chebyshev_rot covers them
    k_chebyshev_dual<R><<<nblocks(s.n, 256), 256, 0, st>>>(s, (R)omega, it, T);
    count_launch(c);
}

template <typename R>
void launch_velocity(avbd_ctx* c, DevState<R>& s, const StepConsts& k, cudaStream_t st) {
    k_velocity<R><<<nblocks(s.n, 256), 256, 0, st>>>(s, (R)(1.0 / k.dt));
    count_launch(c);
}

template <typename R>
void launch_residual(avbd_ctx* c, DevState<R>& s, const StepConsts& k, double* out2, cudaStream_t st,
                     const SceneTol& T) {
    if (out2) cudaMemsetAsync(out2, 0, 2 * sizeof(double), st);
    solve_lanes<MODE_RESIDUAL>(c, s, k, 0, s.n, st, out2, T);
    if (c->dyn) {  // the positional vertices the slab pass skipped
        const uint32_t* list = nullptr;
        unsigned m = 0;
        dyn_positional_list(c, &list, &m);
        if (m) solve_lanes<MODE_RESIDUAL>(c, s, k, 0, m, st, out2, T, list);
    }
}

// ------------------------------------------- per-scene run-to-tolerance
__global__ void k_tol_init(uint8_t* active, uint8_t* cand, double* r2, double* ex, uint32_t* iters, unsigned S,
                           unsigned long long* maxr, uint32_t* it, double* omega, const double* omega_tab,
                           int* n_active) {
    unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) {
        *maxr = 0ull;
        *n_active = (int)S;
        *it = 0;
        if (omega_tab) *omega = omega_tab[0];
    }
    if (s >= S) return;
    active[s] = 1;
    cand[s] = 0;
    r2[s] = r2[S + s] = r2[2 * S + s] = 0;
    ex[s] = ex[S + s] = 0;
    iters[s] = 0;
}

// In-sweep decision of a scene after a sweep: an active scene counts the
// iteration and becomes a candidate when its in-sweep residual is at the
// tolerance.  The in-sweep residual is kept (rin) as the final residual of a
// scene that then stops at the cap without becoming a candidate.
__global__ void k_tol_decide_a(IterArgs A) {
    unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= A.S) return;
    A.cand[s] = 0;
    if (A.active[s]) {
        A.iters[s]++;
        atomicAdd(A.scene_iterations, 1ull);
        const double R = scene_R(A.r2[s], A.m2[s] * A.g2);
        A.rin[s] = R;
        A.cand[s] = R <= A.tol;
    }
    A.r2[s] = 0;
}

// Candidates whose exact residual is at the tolerance stop; so does every
// scene at the iteration cap.  Counts the scenes still iterating.  maxr[0]
// receives the largest final residual of the step's scenes: the exact one
// where it was evaluated in the stopping iteration, else the in-sweep one of
// a capped scene; maxr[1] counts the capped scenes.
__global__ void k_tol_decide_b(IterArgs A) {
    unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= A.S) return;
    if (A.active[s]) {
        bool done = false;
        double R = A.rin[s];
        if (A.cand[s]) {
            R = scene_R(A.ex[s], A.m2[s] * A.g2);
            done = R <= A.tol;
        }
        if (!done && A.iters[s] >= A.max_it) {  // stopped at the cap, unconverged
            done = true;
            atomicAdd(A.maxr + 1, 1ull);
        }
        if (done) {
            A.active[s] = 0;
            atomicMax(A.maxr, ord_enc64(R));
        } else {
            atomicAdd(A.n_active, 1);
        }
    }
    A.cand[s] = 0;
    A.ex[s] = 0;
}

// the run-to-tolerance part of an iteration launch's arguments
static IterArgs tol_args(avbd_ctx* c, double tol, unsigned max_it) {
    IterArgs A = {};
    A.max_it = max_it;
    A.tol = tol;
    A.g2 = c->params.g_accel * c->params.g_accel;
    A.m2 = c->d_scene_mg2;
    A.active = c->d_scene_active;
    A.cand = c->d_scene_cand;
    A.iters = c->d_scene_iters;
    A.r2 = c->d_scene_r2;
    A.ex = c->d_scene_ex;
    A.rin = c->d_scene_rin;
    A.S = c->num_scenes;
    A.scene_iterations = c->d_counters + 1;
    A.maxr = c->d_counters + 2;
    A.n_active = c->d_tol_count;
    return A;
}

void launch_tol_init(avbd_ctx* c, cudaStream_t st) {
    unsigned S = c->num_scenes;
    k_tol_init<<<nblocks(S, 256), 256, 0, st>>>(c->d_scene_active, c->d_scene_cand, c->d_scene_r2, c->d_scene_ex,
                                                c->d_scene_iters, S, c->d_counters + 2, c->d_tol_it, c->d_tol_omega,
                                                c->d_omega_tab, c->d_tol_count);
    count_launch(c);
}

void launch_tol_decide_a(avbd_ctx* c, double tol, cudaStream_t st) {
    k_tol_decide_a<<<nblocks(c->num_scenes, 256), 256, 0, st>>>(tol_args(c, tol, 0));
    count_launch(c);
}

void launch_tol_decide_b(avbd_ctx* c, double tol, unsigned max_it, cudaStream_t st) {
    cudaMemsetAsync(c->d_tol_count, 0, sizeof(int), st);
    k_tol_decide_b<<<nblocks(c->num_scenes, 256), 256, 0, st>>>(tol_args(c, tol, max_it));
    count_launch(c);
}

// One warp per piece: its vertices' lists, filled up to whole rounds.
template <typename RS>
__global__ void k_layout_pieces(TetElems<RS> el, const uint4* slabs, unsigned ncolors, unsigned lanes, uint4* piece,
                                unsigned npieces, StarNb<RS>* pnb, StarTet<RS>* ptet, uint32_t* ploc) {
    const unsigned k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, wl = threadIdx.x & 31u;
    if (k >= npieces) return;
    unsigned col = 0;
    while (col + 1 < ncolors && slabs[col + 1].z <= k) col++;
    const uint4 sl = slabs[col];
    const uint4 h = piece[k];
    const unsigned V = 32 / lanes, gi = (k - sl.z) * V + wl / lanes, lane = wl % lanes;
    const bool live = gi < sl.y;
    const unsigned p = sl.x + min(gi, sl.y - 1);
    const uint2 o0 = el.star[p], o1 = live ? el.star[p + 1] : o0;
    for (unsigned u = 0; u < h.y; u++) {
        const unsigned j = o0.x + lane + u * lanes;
        StarNb<RS> q{};
        q.idx = p;
        if (j < o1.x) q = el.nb[j];
        pnb[h.x + u * 32 + wl] = q;
    }
    for (unsigned u = 0; u < h.w; u++) {
        const unsigned t = o0.y + lane + u * lanes;
        const bool in = t < o1.y;
        ptet[h.z + u * 32 + wl] = in ? el.tet[t] : StarTet<RS>{RS(0), RS(0)};
        ploc[h.z + u * 32 + wl] = in ? el.loc[t] : 0u;
    }
}

template <typename R, typename RS>
static int layout_pieces_t(avbd_ctx* c, TetElems<RS>& el, cudaStream_t st) {
    auto release = [c] {
        for (void* p : c->piece_alloc) cudaFree(p);
        c->piece_alloc.clear();
    };
    release();
    el.piece = nullptr;
    const unsigned lanes = (unsigned)c->lanes;
    if (!el.star || lanes == 2 || c->star_off.empty()) return AVBD_OK;
    const unsigned V = 32 / lanes;
    std::vector<uint4> slabs(c->num_colors), piece;
    size_t nn = 0, nt = 0;
    for (unsigned k = 0; k < c->num_colors; k++) {
        const unsigned b = c->color_begin[k], e = b + c->color_solve[k];
        slabs[k] = make_uint4(b, e - b, (unsigned)piece.size(), 0);
        for (unsigned i = b; i < e; i += V) {
            unsigned mn = 0, mt = 0;
            for (unsigned j = i; j < std::min(i + V, e); j++) {
                mn = std::max(mn, c->star_off[j + 1].x - c->star_off[j].x);
                mt = std::max(mt, c->star_off[j + 1].y - c->star_off[j].y);
            }
            const uint4 h = make_uint4((unsigned)nn, nblocks(mn, lanes), (unsigned)nt, nblocks(mt, lanes));
            piece.push_back(h);
            nn += 32ull * h.y;
            nt += 32ull * h.w;
        }
    }
    if (piece.empty() || nn > UINT32_MAX || nt > UINT32_MAX) return AVBD_OK;  // not laid out: launches per color
    uint4* dp = nullptr;
    StarNb<RS>* dn = nullptr;
    StarTet<RS>* dt = nullptr;
    uint32_t* dl = nullptr;
    auto al = [&](auto** p, size_t bytes) {
        if (cudaMalloc((void**)p, std::max(bytes, (size_t)16)) != cudaSuccess) return false;
        c->piece_alloc.push_back((void*)*p);
        return true;
    };
    if (!al(&dp, sizeof(uint4) * piece.size()) || !al(&dn, sizeof(StarNb<RS>) * nn) ||
        !al(&dt, sizeof(StarTet<RS>) * nt) || !al(&dl, sizeof(uint32_t) * nt)) {
        release();  // no room for a second copy of the lists: not laid out either
        cudaGetLastError();
        return AVBD_OK;
    }
    cudaMemcpyAsync(dp, piece.data(), sizeof(uint4) * piece.size(), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(c->d_slabs, slabs.data(), sizeof(uint4) * slabs.size(), cudaMemcpyHostToDevice, st);
    const unsigned np = (unsigned)piece.size();
    k_layout_pieces<RS><<<nblocks(np, 8), 256, 0, st>>>(el, c->d_slabs, c->num_colors, lanes, dp, np, dn, dt, dl);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return set_error(AVBD_ERR_CUDA, cudaGetErrorString(e));
    el.piece = dp;
    el.pnb = dn;
    el.ptet = dt;
    el.ploc = dl;
    return AVBD_OK;
}
template <typename R>
int layout_pieces(avbd_ctx* c, DevState<R>& s, cudaStream_t st) {
    if (c->solver.precision == AVBD_PRECISION_MIXED) return layout_pieces_t<R>(c, s.el32, st);
    return layout_pieces_t<R>(c, s.el, st);
}

// Blocks of an iteration launch: one per SM, fewer where a color has less
// than a few warps of work for each (a barrier over fewer blocks is cheaper).
static unsigned iterate_blocks(const avbd_ctx* c, unsigned lanes) {
    const unsigned chunks = nblocks(c->max_color_solve, 32 / lanes);
    return std::max(1u, std::min(c->num_sms, nblocks(chunks, ITER_WARPS_MIN)));
}

template <typename P, typename RS, typename HT, int LANES, int FORM>
static bool iterate_launch(avbd_ctx* c, DevState<P>& s, const TetElems<RS>& el, const StepConsts& k, cudaStream_t st,
                           const IterArgs& A) {
    constexpr int THREADS = IterThreads<P, FORM, LANES>::value;
    const bool ground = !c->ground.empty(), tol = A.max_it != 0;
    auto kern = tol ? (ground ? k_iterate<P, RS, HT, LANES, FORM, true, true> : k_iterate<P, RS, HT, LANES, FORM, false, true>)
                    : (ground ? k_iterate<P, RS, HT, LANES, FORM, true, false> : k_iterate<P, RS, HT, LANES, FORM, false, false>);
    constexpr bool PIPE = FORM == FORM_STAR && LANES > 2;
    if (PIPE && !el.piece) return false;
    unsigned smem = FORM == FORM_STAR
                        ? StarStage<P, LANES, THREADS>::bytes(PIPE ? star_rows(el.max_nb, LANES) : el.max_nb)
                        : 0;
    if (tol) smem += 2 * nblocks(A.S, 32) * (unsigned)sizeof(uint32_t);
    if (!stage_smem(kern, smem)) {
        cudaGetLastError();
        return false;
    }
    // whether one block per SM is resident (the grid barrier needs all of
    // them), queried once per lane count and kind of step
    int8_t& fits = c->iterate_fits[tol][LANES == 2 ? 0 : LANES == 4 ? 1 : 2];
    if (fits == 0) {
        int per_sm = 0, coop = 0;
        fits = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) == cudaSuccess && coop &&
                       cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS, smem) == cudaSuccess &&
                       per_sm >= 1
                   ? 1
                   : -1;
        cudaGetLastError();
    }
    if (fits < 0) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(iterate_blocks(c, LANES));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaMemsetAsync(c->d_sweep_sync, 0, 4 * sizeof(unsigned), st);
    // a failed launch is left in the runtime's last error, which the step checks
    cudaLaunchKernelEx(&cfg, kern, s, el, mkc<P>(k), c->d_counters, (const uint32_t*)c->d_scene, A);
    count_launch(c);
    return true;
}

template <typename P, typename RS, typename HT>
static bool iterate_t(avbd_ctx* c, DevState<P>& s, const TetElems<RS>& el, const StepConsts& k, cudaStream_t st,
                      const IterArgs& A) {
    if (el.star) {
        switch (c->lanes) {
            case 2: return iterate_launch<P, RS, HT, 2, FORM_STAR>(c, s, el, k, st, A);
            case 4: return iterate_launch<P, RS, P, 4, FORM_STAR>(c, s, el, k, st, A);
            case 8: return iterate_launch<P, RS, P, 8, FORM_STAR>(c, s, el, k, st, A);
            default: return false;  // not laid out for k_iterate
        }
    }
    // 2 or 8 lanes, the nearer of the context's (launches per color have 4 and 16 too)
    if (c->damping)
        return c->lanes <= 4 ? iterate_launch<P, RS, HT, 2, FORM_DAMP>(c, s, el, k, st, A)
                             : iterate_launch<P, RS, HT, 8, FORM_DAMP>(c, s, el, k, st, A);
    return c->lanes <= 4 ? iterate_launch<P, RS, HT, 2, FORM_REC>(c, s, el, k, st, A)
                         : iterate_launch<P, RS, HT, 8, FORM_REC>(c, s, el, k, st, A);
}
static bool iterate(avbd_ctx* c, DevState<float>& s, const StepConsts& k, cudaStream_t st, const IterArgs& A) {
    return iterate_t<float, float, float>(c, s, s.el, k, st, A);
}
static bool iterate(avbd_ctx* c, DevState<double>& s, const StepConsts& k, cudaStream_t st, const IterArgs& A) {
    if (c->solver.precision == AVBD_PRECISION_MIXED) return iterate_t<double, float, float>(c, s, s.el32, k, st, A);
    return iterate_t<double, double, double>(c, s, s.el, k, st, A);
}

// k_iterate's 12 to 16 warps an SM save launches and passes over small colors;
// k_solve_tet's 24 and more stream large ones better.  ms a step, this launch
// against launches per color, by the vertices of the largest color:
// Star form, to 1e-4, MIXED: 84,000 11.2 and 21.7, 175,000 24.2 and 29.0,
// 326,000 45.5 and 39.0, 1,230,000 165 and 125; FP64: 175,000 38.1 and 33.7;
// FP32: 481,000 46.2 and 49.6, 754,000 68.4 and 73.3.  Fixed iterations: MIXED
// 654,000 10.1 and 10.5, FP32 175,000 equal, FP64 175,000 4.17 and 3.66.
// Records, fixed iterations, FP32: 1,459 0.341 and 0.353, 3,907 0.387 and 0.383,
// 8,985 0.531 and 0.499, 17,231 0.852 and 0.721, 120,691 4.75 and 3.66; random
// points MIXED: 4,436 1.77 and 1.74, 17,744 3.17 and 2.86, 41,228 5.72 and 3.48;
// FP64: 4,436 1.69 and 1.79, 44,360 7.54 and 7.27 (grids 30,523 2.19 and 2.25,
// 241,611 14.7 and 14.0).  Records to tolerance, where a launch per color also
// pays for the decisions: MIXED 481,124 143 and 158, FP64 241,611 103 and 119,
// FP32 481,124 92 and 111.
bool colors_fill_launches(const avbd_ctx* c) {
    const bool tol = c->solver.residual_tolerance > 0;
    if (c->star_nb == 0) return !tol && c->max_color_solve >= (c->solver.precision == AVBD_PRECISION_FP32 ? 4000u : 10000u);
    if (c->solver.precision == AVBD_PRECISION_FP64) return c->max_color_solve >= 130000;
    return tol && c->solver.precision == AVBD_PRECISION_MIXED && c->max_color_solve >= 250000;
}

bool whole_iterations(const avbd_ctx* c) {
    return c->persistent && !c->color_lists && !colors_fill_launches(c) && !c->dyn && c->num_sms != 0 &&
           c->max_color_solve != 0;
}

template <typename R>
bool launch_iterate(avbd_ctx* c, DevState<R>& s, const StepConsts& k, cudaStream_t st, const IterLaunch& L) {
    if (s.no != 0 || !whole_iterations(c)) return false;
    IterArgs A = {};
    if (L.tol > 0) {
        A = tol_args(c, L.tol, L.max_it);
        if (L.loop) {
            A.it_dev = c->d_tol_it;
            A.loop = *L.loop;
            A.has_loop = true;
            A.launches = c->d_counters + 5;
        }
    }
    A.slabs = c->d_slabs;
    A.ncolors = c->num_colors;
    A.omega = c->d_omega_tab;
    A.it0 = L.it0;
    A.n = L.n;
    A.sync = c->d_sweep_sync;
    A.sweep_only = L.sweep_only;
    return iterate(c, s, k, st, A);
}

// End of one iteration of the device-driven loop: counts it and continues the
// while node while scenes are still iterating.  iters of a scene reach max_it
// within max_it iterations, so n_active is 0 by then; the index bound stops
// the loop at max_it in any case.  Also counts the body's kernel launches.
__global__ void k_tol_loop_next(cudaGraphConditionalHandle h, const int* n_active, uint32_t* it,
                                const double* omega_tab, double* omega, unsigned max_it,
                                unsigned long long body_launches, unsigned long long* launches) {
    const uint32_t i = *it + 1;
    *it = i;
    *launches += body_launches;
    const bool more = *n_active > 0 && i < max_it;
    if (more) *omega = omega_tab[i];
    cudaGraphSetConditional(h, more ? 1u : 0u);
}

void launch_tol_loop_next(avbd_ctx* c, cudaGraphConditionalHandle h, unsigned max_it, unsigned body_launches,
                          cudaStream_t st) {
    k_tol_loop_next<<<1, 1, 0, st>>>(h, c->d_tol_count, c->d_tol_it, c->d_omega_tab, c->d_tol_omega, max_it,
                                     body_launches + 1ull, c->d_counters + 5);
}

__global__ void k_iter_set(uint32_t* it, double* omega, const double* omega_tab) {
    *it = 0;
    *omega = omega_tab[0];
}
__global__ void k_iter_next(uint32_t* it, double* omega, const double* omega_tab, unsigned n) {
    const uint32_t i = *it + 1;
    *it = i;
    if (i < n) *omega = omega_tab[i];
}
void launch_iter_set(avbd_ctx* c, cudaStream_t st) {
    k_iter_set<<<1, 1, 0, st>>>(c->d_tol_it, c->d_tol_omega, c->d_omega_tab);
    count_launch(c);
}
void launch_iter_next(avbd_ctx* c, unsigned n, cudaStream_t st) {
    k_iter_next<<<1, 1, 0, st>>>(c->d_tol_it, c->d_tol_omega, c->d_omega_tab, n);
    count_launch(c);
}

template <typename R>
void launch_debug_block(avbd_ctx* c, DevState<R>& s, const StepConsts& k, unsigned p, double* out, cudaStream_t st) {
    solve_lanes<MODE_DEBUG>(c, s, k, p, 1, st, out, SceneTol());
}

// warm-start features of every solved tet vertex at the current iterate,
// one 64-byte BF16 row per internal vertex
template <typename R>
void launch_features(avbd_ctx* c, DevState<R>& s, const StepConsts& k, void* feat, const float* prev,
                     cudaStream_t st) {
    c->ws_prev_arg = prev;
    solve_lanes<MODE_FEATURES>(c, s, k, 0, s.n, st, reinterpret_cast<double*>(feat), SceneTol());
    c->ws_prev_arg = nullptr;
}

// copy of the solved vertices' warm-start positions (x0)
template <typename R>
__global__ void k_ws_save(const DevState<R> s, typename Vec4Of<R>::T* x0) {
    unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < s.n) x0[p] = s.x[p];
}

// target row (x_end - x0) / s, column 3 = 1 for solved tet vertices, else 0
template <typename R>
__global__ void k_ws_target(const DevState<R> s, const typename Vec4Of<R>::T* x0, float inv_s, float4* t) {
    unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n) return;
    if (s.flags[p] & (VF_FIXED | VF_ORIENTED)) {
        t[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    typename Vec4Of<R>::T a = s.x[p], b = x0[p];
    t[p] = make_float4((float)(a.x - b.x) * inv_s, (float)(a.y - b.y) * inv_s, (float)(a.z - b.z) * inv_s, 1.f);
}

template <typename R>
void launch_ws_save(avbd_ctx* c, DevState<R>& s, void* x0, cudaStream_t st) {
    k_ws_save<R><<<nblocks(s.n, 256), 256, 0, st>>>(s, reinterpret_cast<typename Vec4Of<R>::T*>(x0));
    count_launch(c);
}

template <typename R>
void launch_ws_target(avbd_ctx* c, DevState<R>& s, const void* x0, double inv_s, float* t, cudaStream_t st) {
    k_ws_target<R><<<nblocks(s.n, 256), 256, 0, st>>>(s, reinterpret_cast<const typename Vec4Of<R>::T*>(x0),
                                                       (float)inv_s, reinterpret_cast<float4*>(t));
    count_launch(c);
}

template <typename R>
void launch_load_positions(DevState<R>& s, const double* src, const uint32_t* inv_map, unsigned first, unsigned n,
                           int mode, cudaStream_t st) {
    if (n == 0) return;
    k_load<R><<<nblocks(n, 256), 256, 0, st>>>(s, src, inv_map, first, n, mode);
}

template <typename R>
void launch_store_vec(const DevState<R>& s, int which, double* dst, const uint32_t* inv_map, unsigned n,
                      cudaStream_t st) {
    if (n == 0) return;
    k_store<R><<<nblocks(n, 256), 256, 0, st>>>(s, which, dst, inv_map, 0, n);
}

#define INST(R)                                                                                                  \
    template void launch_begin_step<R>(avbd_ctx*, DevState<R>&, const StepConsts&, cudaStream_t);               \
    template void launch_tet_eprev<R>(avbd_ctx*, DevState<R>&, const StepConsts&, cudaStream_t);                \
    template void launch_solve_color<R>(avbd_ctx*, DevState<R>&, const StepConsts&, unsigned, unsigned,         \
                                        cudaStream_t, const SceneTol&, const uint32_t*, const uint4*, unsigned); \
    template bool launch_iterate<R>(avbd_ctx*, DevState<R>&, const StepConsts&, cudaStream_t, const IterLaunch&); \
    template int layout_pieces<R>(avbd_ctx*, DevState<R>&, cudaStream_t);                                        \
    template void launch_chebyshev_dual<R>(avbd_ctx*, DevState<R>&, const StepConsts&, double, unsigned, cudaStream_t,    \
                                           const SceneTol&);                                                    \
    template void launch_velocity<R>(avbd_ctx*, DevState<R>&, const StepConsts&, cudaStream_t);                 \
    template void launch_residual<R>(avbd_ctx*, DevState<R>&, const StepConsts&, double*, cudaStream_t,         \
                                     const SceneTol&);                                                          \
    template void launch_debug_block<R>(avbd_ctx*, DevState<R>&, const StepConsts&, unsigned, double*,          \
                                        cudaStream_t);                                                          \
    template void launch_features<R>(avbd_ctx*, DevState<R>&, const StepConsts&, void*, const float*,           \
                                     cudaStream_t);                                                             \
    template void launch_ws_save<R>(avbd_ctx*, DevState<R>&, void*, cudaStream_t);                               \
    template void launch_ws_target<R>(avbd_ctx*, DevState<R>&, const void*, double, float*, cudaStream_t);       \
    template void launch_load_positions<R>(DevState<R>&, const double*, const uint32_t*, unsigned, unsigned, int, \
                                           cudaStream_t);                                                       \
    template void launch_store_vec<R>(const DevState<R>&, int, double*, const uint32_t*, unsigned, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace avbd
