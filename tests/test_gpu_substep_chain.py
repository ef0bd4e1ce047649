"""The binning, block sort and placement chain of a substep at the edges of its tiles: particle counts
around the threads of a block and the particles of a thread, masked particles, scenes with a slicer
(whose records and cut masks are rebuilt every substep) and batches that mix both.  Calls of several
substeps (bins and records carried from substep to substep) and single steps agree with the FP64
oracle within the parity bar and with each other."""
import numpy as np
import pytest

from conftest import cuda_available
from gpu_helpers import rel_pos_err

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
import oracle_py as op  # noqa: E402
from crmpm_b200 import scenes  # noqa: E402

KEYS = ("pos_mass", "vel", "mat_params", "mat_type", "mask")


def _scene(kind, n):
    sc = scenes.cube_drop() if kind == "plane" else scenes.contact_scene(kind)
    if kind == "plane":
        sc.vel[:, :3] = (0.3, -1.0, 0.2)
    pick = np.linspace(0, sc.n - 1, n).astype(int)  # spread over the body: many thinly filled blocks
    for k in KEYS:
        setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[pick]))
    sc.mask[::7] = 0 if n > 7 else 1
    sc.iterations = 10  # one value for a batch (no part in MLS-MPM)
    return sc


def _check(got, sc, steps):
    o = op.PortOracle(sc, 64)
    o.compute_initial_data()
    o.step(steps)
    ref = o.state()
    assert rel_pos_err(got["x"], ref["x"], sc.pos_mass[:, :3], sc.cell_size) < 1e-4
    np.testing.assert_allclose(got["v"], ref["v"], atol=1e-3 * max(np.abs(ref["v"]).max(), 1e-6))


@pytest.mark.parametrize("kind", ["plane", "quad_slicer"])
@pytest.mark.parametrize("n", [1, 7, 128, 255, 257, 1023, 1025, 3073])
def test_call_lengths_agree(kind, n):
    sc = _scene(kind, n)
    a, b = cb.DeviceScene(sc), cb.DeviceScene(sc)
    a.step(5)
    b.step(5, graph=False)
    sa, sb = a.state(), b.state()
    _check(sa, sc, 5)
    assert rel_pos_err(sa["x"], sb["x"], sc.pos_mass[:, :3], sc.cell_size) < 1e-5
    assert a.solver.grid_stats()["num_sorted"] == int(sc.mask.sum())
    a.step(3)  # a second call starts from clean counters
    _check(a.state(), sc, 8)


def test_batch_of_scenes_with_and_without_slicer():
    parts = [_scene("plane", 257), _scene("quad_slicer", 1025), _scene("plane", 31), _scene("quad_slicer", 513)]
    b = cb.DeviceBatch(parts)
    b.step(4)
    st = b.state()
    for s, sc in enumerate(parts):
        _check(b.scene_state(s, st), sc, 4)
    assert b.solver.grid_stats()["num_sorted"] == sum(int(sc.mask.sum()) for sc in parts)


@pytest.mark.parametrize("cells,ppc", [(15, 8), (16, 8), (23, 8), (24, 8), (4, 40), (12, 40)])
@pytest.mark.parametrize("solver", ["mls", "standard", "deterministic"])
def test_threads_per_cell(cells, ppc, solver):
    """Both sides of the particle counts at which a cell gets 4, 2 and 1 threads (27000 / 32768, 97336 /
    110592), and cells fuller than the threads' runs."""
    sc = scenes.cube_drop(side=cells * 0.02, cell=0.02, ppc=ppc,
                          solver=scenes.SOLVER_STANDARD if solver == "standard" else scenes.SOLVER_MLS)
    sc.pos_mass[:, 1] -= np.float32(0.5 - cells * 0.01 - 0.01)
    sc.vel[:, :3] = (0.2, -1.0, 0.1)
    g = cb.DeviceScene(sc, compute_initial=solver != "deterministic")
    if solver == "deterministic":
        g.solver.set_option(cb.OPT_DETERMINISTIC, 1)
        g.compute_initial_data()
    g.step(4)
    _check(g.state(), sc, 4)
