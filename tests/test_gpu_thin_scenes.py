"""The cell accumulation where few particles lie in many blocks: the 64-thread groups of a CTA then take
blocks of their own instead of sharing one.  Both sides of the number of blocks at which they do,
cells fuller than a group's run, batches on both sides of the particle counts at which a cell gets 4, 2
and 1 threads, against the FP64 oracle; and the time of a thin scene beside a larger one."""
import statistics

import numpy as np
import pytest

from conftest import cuda_available
from gpu_helpers import rel_pos_err

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
import oracle_py as op  # noqa: E402
from crmpm_b200 import scenes  # noqa: E402

SOLVERS = {"mls": scenes.SOLVER_MLS, "deterministic": scenes.SOLVER_MLS, "standard": scenes.SOLVER_STANDARD,
           "pb": scenes.SOLVER_PB}


def _thin(solver, cells, ppc, seed=1001):
    sc = scenes.cube_drop(seed=seed, side=cells * 0.02, cell=0.02, ppc=ppc, solver=SOLVERS[solver], dt=1e-4)
    sc.vel[:, :3] = (0.2, -1.0, 0.1)
    sc.iterations = 3
    if solver == "pb":
        sc.mat_params[:, :2] = (1.0, 0.9)
    return sc


def _clustered(solver, blocks, per_cell):
    """One full cell in each of blocks^3 blocks of 4x4x4 cells, and one particle in a cell beside it."""
    sc = _thin(solver, blocks, per_cell + 1)
    cell = sc.pos_mass[:, :3].copy()
    cell = np.floor((cell - cell.min(axis=0)) / 0.02 + 1e-3)
    inside = sc.pos_mass[:, :3] - sc.pos_mass[:, :3].min(axis=0) - cell * 0.02
    sc.pos_mass[:, :3] = np.clip(inside, 1e-3, 0.019) + cell * 0.08 + (-0.04 * blocks, 0.1, -0.04 * blocks)
    sc.pos_mass[::per_cell + 1, 0] += np.float32(0.02)
    return sc


def _gpu(sc, solver):
    g = (cb.DeviceBatch if isinstance(sc, list) else cb.DeviceScene)(sc, compute_initial=solver != "deterministic")
    if solver == "deterministic":
        g.solver.set_option(cb.OPT_DETERMINISTIC, 1)
        g.compute_initial_data()
    return g


def _check(got, sc, steps):
    """Positions within 1e-4 of max(displacement, dx) of FP64, or twice the float32 oracle's own departure."""
    ref, ref32 = op.PortOracle(sc, 64), op.PortOracle(sc, 32)
    for o in (ref, ref32):
        o.compute_initial_data()
        o.step(steps)
    a, b = ref.state(), ref32.state()
    x0 = sc.pos_mass[:, :3]
    assert rel_pos_err(got["x"], a["x"], x0, sc.cell_size) <= max(1e-4, 2 * rel_pos_err(b["x"], a["x"], x0, sc.cell_size))
    dv = np.abs(b["v"] - a["v"]).max()
    assert np.abs(got["v"] - a["v"]).max() <= max(1e-3 * np.abs(a["v"]).max(), 2 * dv)


@pytest.mark.parametrize("cells,ppc", [(15, 1), (20, 1), (30, 1), (34, 1), (26, 2), (28, 4)])
@pytest.mark.parametrize("solver", sorted(SOLVERS))
def test_blocks_of_their_own(solver, cells, ppc):
    sc = _thin(solver, cells, ppc)
    g = _gpu(sc, solver)
    g.step(3)
    _check(g.state(), sc, 3)


@pytest.mark.parametrize("blocks,per_cell", [(5, 40), (6, 40), (7, 60), (9, 45)])
@pytest.mark.parametrize("solver", sorted(SOLVERS))
def test_full_cells_in_many_blocks(solver, blocks, per_cell):
    sc = _clustered(solver, blocks, per_cell)
    g = _gpu(sc, solver)
    g.step(3)
    assert g.solver.grid_stats()["active_blocks"] >= blocks ** 3
    _check(g.state(), sc, 3)


@pytest.mark.parametrize("num,cells,ppc", [(4, 7, 8), (4, 14, 1), (5, 14, 1), (17, 14, 1), (18, 14, 1)])
@pytest.mark.parametrize("solver", sorted(SOLVERS))
def test_batches(solver, num, cells, ppc):
    parts = [_thin(solver, cells, ppc, seed=1001 + k) for k in range(num)]
    b = _gpu(parts, solver)
    b.step(3)
    st = b.state()
    for s in (0, num // 2, num - 1):
        _check(b.scene_state(s, st), parts[s], 3)


@pytest.mark.parametrize("solver", ["standard", "pb"])
def test_a_thin_scene_is_no_slower_than_a_larger_one(solver):
    """27000 particles in 716 blocks and 32768 in some 730, both one per cell: the smaller scene takes no
    longer than a tenth above the larger one's time."""
    import torch

    pair = [cb.DeviceScene(_thin(solver, cells, 1)) for cells in (30, 32)]
    took = ([], [])
    for rep in range(12):
        for g, out in zip(pair, took):
            start, stop = torch.cuda.Event(True), torch.cuda.Event(True)
            torch.cuda.synchronize()
            start.record(g.stream)
            g.step(10)
            stop.record(g.stream)
            torch.cuda.synchronize()
            out.append(start.elapsed_time(stop))
    small, large = (statistics.median(t[2:]) for t in took)
    print(f"{solver}: {1e3 * small:.0f} us, {1e3 * large:.0f} us")
    assert small <= 1.1 * large
