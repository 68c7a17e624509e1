"""The star form of the tet solve and the iteration launch at their edges,
against the FP64 oracle: every lane count of the launch, scenes that stop in
different iterations, vertices with more neighbours than a piece prefetches
(16) or the star form takes (64: the context falls back to the records),
particles without any tet.

Tolerances are those of the parity tests: the FP64 engine differs from the
oracle by summation order (1e-9 of the bounding-box diagonal), the mixed one
by its FP32 element constants (1e-6), FP32 without contact by 1e-5.
"""
import threading

import numpy as np
import pytest

from avbd_b200 import Context, scenes

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-9, "mixed": 1e-6, "fp32": 1e-5}


def _pair(oracle_lib, sc, precision, **kw):
    e = Context()
    sc.load(e, precision=precision, **kw)
    e.finalize()
    o = oracle_lib.Oracle()
    sc.load(o, **kw)
    o.finalize()
    return e, o


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("whole", [1, 0])
def test_lane_counts_to_tolerance(oracle_lib, monkeypatch, whole, lanes, precision):
    """Uneven scenes of odd sizes; they stop in different iterations, so the
    launch changes from contiguous to dealt pieces on the way.  whole 0: the
    launches per color that large colors take."""
    monkeypatch.setenv("AVBD_PERSISTENT", str(whole))
    monkeypatch.setenv("AVBD_LANES", str(lanes))
    sc = scenes.batched_cubes(num_scenes=7, seed=9, n_min=2, n_max=7)
    e, o = _pair(oracle_lib, sc, precision, residual_tolerance=1e-4, max_iters=120)
    stopped = set()
    for step in range(4):
        e.step(1)
        o.step(1)
        ie, io = e.scene_iterations().astype(int), o.scene_iterations().astype(int)
        assert np.abs(ie - io).max() <= 2, (step, ie, io)
        stopped |= set(io.tolist())
        err = np.abs(e.positions() - o.positions()).max() / sc.bbox_diagonal()
        assert err <= TOL[precision], (step, err)
    assert len(stopped) > 2  # the scenes did stop at different times


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("lanes", [1, 4, 8, 16])
def test_lane_counts_fixed_iterations(oracle_lib, monkeypatch, lanes, precision):
    monkeypatch.setenv("AVBD_LANES", str(lanes))
    sc = scenes.cube_fixed_bottom(5, iters=7)
    e, o = _pair(oracle_lib, sc, precision)
    e.step(6)
    o.step(6)
    assert np.abs(e.positions() - o.positions()).max() / sc.bbox_diagonal() <= TOL[precision]


def fan(k: int) -> scenes.Scene:
    """k tets around one edge: its ends have k + 1 neighbours."""
    sc = scenes.Scene(name=f"fan{k}", dt=1.0 / 60.0, solver_iters=10)
    a = np.arange(k) * 2 * np.pi / k
    X = np.concatenate([[[0.0, 0.5, 0.0], [0.0, 1.1, 0.0]],
                        np.stack([np.cos(a), 0.6 + 0.05 * np.sin(3 * a), np.sin(a)], axis=1)])
    i = np.arange(k)
    T = np.stack([np.zeros(k, int), np.ones(k, int), 2 + i, 2 + (i + 1) % k], axis=1)
    Q, V, lam, mu, m = scenes.tet_setup(X, T, 1e5, 0.4, 1000.0)
    sc.record("add_particles", X, m)
    sc.record("add_neo_hookean", T, np.full(k, lam), np.full(k, mu), np.zeros(k), Q.reshape(-1, 9), V)
    sc.record("set_fixed", [2, 3], np.ones(2, np.uint8))
    sc.meta["bbox_diagonal"] = 2.9
    return sc


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("k", [15, 16, 40, 63, 64, 90])
def test_many_neighbours(oracle_lib, k, precision):
    sc = fan(k)
    e, o = _pair(oracle_lib, sc, precision)
    e.step(3)
    o.step(3)
    assert np.abs(e.positions() - o.positions()).max() / sc.bbox_diagonal() <= TOL[precision]
    # the blocks of the edge's ends and of a ring vertex
    tol = 2e-4 if precision == "fp32" else 1e-5 if precision == "mixed" else 1e-7
    o.set_positions_raw(0, e.positions())
    for p in (0, 1, 4):
        G, H = e.debug_block(p)
        Go, Ho = o.debug_block(p)[:2]
        assert np.abs(H - Ho).max() <= tol * np.abs(Ho).max()
        if precision == "fp64":
            assert np.abs(G - Go).max() <= 1e-6 * max(1.0, np.abs(Go).max())


def test_particles_without_tets(oracle_lib):
    sc = scenes.Scene(name="free", dt=1.0 / 60.0, solver_iters=5)
    X = np.random.default_rng(3).uniform(0.01, 1.0, size=(37, 3))
    m = np.linspace(0.5, 2.0, 37)
    sc.record("add_particles", X, m)
    sc.record("add_ground_collision", np.arange(37), m / sc.dt ** 2, np.full(37, 0.4), np.full(37, 0.2))
    e, o = _pair(oracle_lib, sc, "fp64")
    e.step(30)
    o.step(30)
    assert np.abs(e.positions() - o.positions()).max() <= 1e-9


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("twice", [(9, 9, 2, 5), (2, 9, 9, 0), (7, 3, 6, 7), (1, 4, 1, 8)])
def test_tet_with_a_repeated_vertex(oracle_lib, twice, precision):
    """Accepted by the entry points: the edge between the two is zero.  The
    repeated vertex is the largest, the smallest or one between its
    neighbours.  Blocks as in test_many_neighbours."""
    sc = fan(8)
    Q = np.array([[1.1, 0.2, -0.3, 0.1, 0.9, 0.2, -0.2, 0.3, 1.3]])
    sc.record("add_neo_hookean", np.array([twice]), np.array([1e5]), np.array([4e4]), np.zeros(1), Q, np.array([0.02]))
    e, o = _pair(oracle_lib, sc, precision)
    e.step(2)
    X = e.positions()
    assert np.isfinite(X).all()
    o.set_positions_raw(0, X)
    tol = 2e-4 if precision == "fp32" else 1e-5 if precision == "mixed" else 1e-7
    for p in sorted({0, 1} | set(twice) - {2, 3}):
        G, H = e.debug_block(p)
        Go, Ho = o.debug_block(p)[:2]
        assert np.abs(H - Ho).max() <= tol * np.abs(Ho).max()
        if precision == "fp64":
            assert np.abs(G - Go).max() <= 1e-6 * max(1.0, np.abs(Go).max())


@pytest.mark.parametrize("whole", [1, 0])
def test_tolerance_without_gravity(oracle_lib, monkeypatch, whole):
    """The residual is then the absolute force (its scale, the weight, is 0):
    scenes stop where the oracle's do, not at the cap."""
    monkeypatch.setenv("AVBD_PERSISTENT", str(whole))
    sc = scenes.batched_cubes(num_scenes=5, seed=9, n_min=2, n_max=5)
    sc.g_accel = 0.0
    e, o = _pair(oracle_lib, sc, "fp64", residual_tolerance=1e-2, max_iters=120)
    V = np.random.default_rng(3).uniform(-0.2, 0.2, size=e.positions().shape)
    e.set_velocities(0, V)
    o.set_velocities(0, V)
    for step in range(3):
        e.step(1)
        o.step(1)
        ie, io = e.scene_iterations().astype(int), o.scene_iterations().astype(int)
        assert io.max() < 100 and np.abs(ie - io).max() <= 2, (step, ie, io)
        assert np.abs(e.positions() - o.positions()).max() / sc.bbox_diagonal() <= TOL["fp64"]


@pytest.mark.parametrize("whole", [1, 0])
def test_contexts_of_different_valence_on_two_threads(monkeypatch, whole):
    """Contexts are independent: while one host thread steps a context, another
    steps one whose staging of neighbours takes less shared memory (both more
    than the 48 KB a kernel has without opting in).  Every launch is a call of
    its own (no graph), so that the two meet often; fixed iterations are
    deterministic, so each ends where it ends alone."""
    monkeypatch.setenv("AVBD_PERSISTENT", str(whole))
    monkeypatch.setenv("AVBD_GRAPH", "0")
    sizes, steps = (60, 52), 400

    def context(k):
        e = Context()
        fan(k).load(e, precision="fp64")
        e.finalize()
        return e

    def run(e, errors):
        try:
            for _ in range(steps):
                e.step(1)
            e.synchronize()
        except Exception as ex:
            errors.append(repr(ex))

    alone = []
    for k in sizes:
        e = context(k)
        errors = []
        run(e, errors)
        assert not errors
        alone.append(e.positions())
        e.close()
    both = [context(k) for k in sizes]
    errors = []
    threads = [threading.Thread(target=run, args=(e, errors)) for e in both]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for e, X in zip(both, alone):
        assert np.array_equal(e.positions(), X)
        e.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("lanes", [2, 4, 8, 16])
@pytest.mark.parametrize("whole", [1, 0])
def test_record_lane_counts(oracle_lib, monkeypatch, whole, lanes, precision):
    """Damped tets (records) with each lane count of the launches per color; the
    iteration launch takes 2 or 8."""
    monkeypatch.setenv("AVBD_PERSISTENT", str(whole))
    monkeypatch.setenv("AVBD_LANES", str(lanes))
    sc = scenes.Scene(name="damped", dt=1.0 / 60.0, solver_iters=7)
    scenes.add_tet_cube(sc, 5, E=1e5, nu=0.45, density=1000.0, fix_bottom=True, kd=5.0)
    e, o = _pair(oracle_lib, sc, precision)
    e.step(6)
    o.step(6)
    assert np.abs(e.positions() - o.positions()).max() / sc.bbox_diagonal() <= TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
def test_lane_choice_of_large_colors_with_many_neighbours(precision):
    """21,600 vertices a color (their lane count is timed), hubs of 21
    neighbours: whatever is chosen, the iterations stay one launch, and every
    scene does what it does alone (other lane counts: other sums)."""
    k, copies = 20, 2400
    one = fan(k)
    (_, (X, m), _), (_, (T, lam, mu, kd, Q, V), _), (_, (held, flags), _) = one.calls
    many = scenes.Scene(name="fans", dt=one.dt, solver_iters=one.solver_iters)
    for s in range(copies):
        if s:
            many.record("begin_scene")
        many.record("add_particles", X, m)
        many.record("add_neo_hookean", T + s * len(X), lam, mu, kd, Q, V)
        many.record("set_fixed", np.asarray(held) + s * len(X), flags)
    e = Context()
    many.load(e, precision=precision)
    e.finalize()
    before = e.stats()["kernel_launches"]
    e.step(1)
    assert e.stats()["kernel_launches"] - before <= 4
    e.step(2)
    a = Context()
    one.load(a, precision=precision)
    a.finalize()
    a.step(3)
    P, A = e.positions().reshape(copies, len(X), 3), a.positions()
    assert np.abs(P - A).max() / one.bbox_diagonal() <= TOL[precision]


def test_route_of_large_record_contexts_follows_the_solver():
    """Damped FP32 colors of some 4,900 vertices: launches per color for a fixed
    number of iterations, the iteration launch to a tolerance, also when the
    solver is set after finalize."""
    sc = scenes.Scene(name="damped", dt=1.0 / 60.0, solver_iters=6)
    scenes.add_tet_cube(sc, 26, E=1e5, nu=0.45, density=1000.0, fix_bottom=True, kd=5.0)
    e = Context()
    sc.load(e, precision="fp32")
    e.finalize()
    colors = e.stats()["num_colors"]

    def launches():
        before = e.stats()["kernel_launches"]
        e.step(1)
        e.synchronize()
        return e.stats()["kernel_launches"] - before

    fixed = launches()
    assert fixed >= 6 * colors
    e.set_solver(6, sc.iter_acceleration, 1e-12, 32, "fp32")  # not reached: 32 iterations
    assert launches() < 32
    e.set_solver(6, sc.iter_acceleration, 0.0, 0, "fp32")
    assert launches() == fixed
    assert np.isfinite(e.positions()).all()
