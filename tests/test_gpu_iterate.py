"""The iteration launch in the forms contexts take by default (4 and 8 threads
a vertex, pieces loaded ahead across the barrier), from the step's graph and
from host launches: its agreement with launches per color, and leaving at a
barrier whose wait runs out, with pieces on their way.
"""
import numpy as np
import pytest

from avbd_b200 import Context, _lib, scenes
from avbd_b200._lib import AvbdError

pytestmark = pytest.mark.gpu

ERR_TIMEOUT = 6


def _ctx(monkeypatch, sc, whole, lanes, graph, tol, precision="fp64"):
    monkeypatch.setenv("AVBD_PERSISTENT", str(whole))
    monkeypatch.setenv("AVBD_GRAPH", str(graph))
    if lanes:
        monkeypatch.setenv("AVBD_LANES", str(lanes))
    else:
        monkeypatch.delenv("AVBD_LANES", raising=False)
    e = Context()
    sc.load(e, residual_tolerance=tol, max_iters=100, precision=precision)
    e.finalize()
    return e


@pytest.mark.parametrize("graph", [1, 0])
@pytest.mark.parametrize("lanes", [None, 4, 8])
@pytest.mark.parametrize("tol", [1e-4, 0.0])
def test_matches_launches_per_color(monkeypatch, tol, lanes, graph):
    """FP64, where the forms differ by summation order alone: 1e-9 of the
    bounding box as against the oracle, and a stop decision on the tolerance
    may fall an iteration apart (then the positions differ by what the
    tolerance allows, so the comparison starts again from the same state)."""
    sc = scenes.batched_cubes(num_scenes=1024, seed=0, scene_ids=range(12))
    a = _ctx(monkeypatch, sc, 0, lanes, graph, tol)
    b = _ctx(monkeypatch, sc, 1, lanes, graph, tol)
    for step in range(3):
        la, lb = a.stats()["kernel_launches"], b.stats()["kernel_launches"]
        a.step(1)
        b.step(1)
        assert b.stats()["kernel_launches"] - lb < a.stats()["kernel_launches"] - la
        if tol and not (a.scene_iterations() == b.scene_iterations()).all():
            assert np.abs(a.scene_iterations().astype(int) - b.scene_iterations().astype(int)).max() <= 1
            break
        assert np.abs(a.positions() - b.positions()).max() / sc.bbox_diagonal() <= 1e-9, step
    a.close()
    b.close()


@pytest.mark.parametrize("graph", [1, 0])
@pytest.mark.parametrize("lanes", [None, 4])
@pytest.mark.parametrize("precision,tol", [("mixed", 1e-4), ("fp32", 0.0)])
def test_barrier_timeout_is_reported(monkeypatch, precision, tol, lanes, graph):
    """With a wait limit of 0 every block but the last to arrive gives up; the
    step reports it and the context steps normally afterwards."""
    sc = scenes.batched_cubes(num_scenes=1024, seed=0, scene_ids=range(12))
    e = _ctx(monkeypatch, sc, 1, lanes, graph, tol, precision)
    e.step(1)
    x0, v0 = e.positions(), e.velocities()
    L = _lib.load()
    try:
        assert L.avbd_debug_set_wait_limit(0, 0) == 0
        with pytest.raises(AvbdError) as ex:
            e.step(1)
            e.synchronize()
        assert ex.value.code == ERR_TIMEOUT
    finally:
        assert L.avbd_debug_set_wait_limit(0, _lib.DEFAULT_WAIT_POLLS) == 0
    e.set_state(x0, v0)
    e.step(2)
    e.synchronize()
    assert np.isfinite(e.positions()).all()
    e.close()


def test_profiled_bytes_of_the_fused_iteration():
    """Beyond the sweep an iteration of the streamed star form moves a history
    read, a history write and a second position (32 bytes each in MIXED) per
    solved vertex; fixed ones have none, ground duals change in place."""
    sc = scenes.Scene(name="cube", dt=1.0 / 60.0, solver_iters=5)
    scenes.add_tet_cube(sc, 6, fix_bottom=True, ground=True)
    e = Context()
    sc.load(e, precision="mixed", residual_tolerance=1e-12, max_iters=1)
    e.finalize()
    sweep = e.profile_solve(1)[1]
    _, step, launches, iterations = e.profile_step()
    assert (launches, iterations) == (1, 1)
    solved = 7 ** 3 - 7 ** 2
    assert step - sweep == pytest.approx(3 * 32 * solved)
    e.close()
