"""Slicer cut masks of MLS-MPM substeps as CrB200SolverCopyCutMasks hands them out: every particle has
one, zero for particles that take no part and in scenes without a slicer."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
import oracle_py as op  # noqa: E402
from crmpm_b200 import scenes  # noqa: E402


def _scene(kind, n=1025):
    sc = scenes.contact_scene(kind)
    pick = np.linspace(0, sc.n - 1, n).astype(int)
    for k in ("pos_mass", "vel", "mat_params", "mat_type", "mask"):
        setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[pick]))
    return sc


def _leave_masks(cls, *args):
    """A solver of the same sizes, all of its scenes cut, that is gone again: a buffer that the next solver
    takes and does not write holds its masks."""
    g = cls(*args)
    g.step(1)
    assert g.cut_masks().any()
    g.sync()


def _expected(sc, x):
    """The oracle's masks (single precision, reference order) at positions x; zero where masked out."""
    o = op.PortOracle(sc, 32)
    o.set_state(x=x.astype(np.float64))
    return np.where(sc.mask != 0, o.cut_masks(), 0).astype(np.uint32)


def _inputs_of_last_substep(make, calls):
    """Positions the last substep of the calls starts from: the same substeps but the last, deterministic."""
    g = make()
    for c in calls[:-1] + ([calls[-1] - 1] if calls[-1] > 1 else []):
        g.step(c)
    return g.state()["x"]


def _deterministic(make):
    def run():
        g = make()
        g.solver.set_option(cb.OPT_DETERMINISTIC, 1)
        g.compute_initial_data()
        return g
    return run


@pytest.mark.parametrize("calls", [[1], [4], [2, 3]])
def test_scene_with_masked_particles(calls):
    sc = _scene("quad_slicer")
    sc.mask[::3] = 0
    make = _deterministic(lambda: cb.DeviceScene(sc, compute_initial=False))
    exp = _expected(sc, _inputs_of_last_substep(make, calls))
    assert exp.any()
    _leave_masks(cb.DeviceScene, _scene("quad_slicer"))
    g = make()
    for c in calls:
        g.step(c)
    np.testing.assert_array_equal(g.cut_masks(), exp)


def test_particles_that_drop_out_between_calls():
    import torch

    sc = _scene("quad_slicer")
    g = cb.DeviceScene(sc)
    g.step(2)
    before = g.cut_masks()
    assert before[::2].any() and before[1::4].any()
    off = sc.mask.copy()
    off[::2] = 0
    g.mask[:sc.n] = torch.from_numpy(off).to(g.device)
    g.pos[1:sc.n:4, 0] = float("nan")
    torch.cuda.synchronize()
    g.step(1)
    masks = g.cut_masks()
    assert not masks[::2].any() and not masks[1::4].any() and masks[3::4].any()


@pytest.mark.parametrize("calls", [[1], [4], [2, 3]])
@pytest.mark.parametrize("kinds", [("quad_slicer",), ("box", "sphere"), ("sphere", "quad_slicer", "box", "quad_slicer")])
def test_batches(kinds, calls):
    sizes = (1025, 513, 257, 769)
    parts = [_scene(k, n) for k, n in zip(kinds, sizes)]
    for sc in parts:
        sc.mask[::5] = 0
    make = _deterministic(lambda: cb.DeviceBatch(parts, compute_initial=False))
    x = _inputs_of_last_substep(make, calls)
    _leave_masks(cb.DeviceBatch, [_scene("quad_slicer", n) for n in sizes[:len(parts)]])
    b = make()
    for c in calls:
        b.step(c)
    masks = b.cut_masks()
    for s, sc in enumerate(parts):
        got = masks[b.batch.slice(s)]
        if kinds[s] == "quad_slicer":
            exp = _expected(sc, x[b.batch.slice(s)])
            assert exp.any()
            np.testing.assert_array_equal(got, exp)
        else:
            assert not got.any()


def test_batch_scenes_that_lose_their_slicer_or_particles():
    import torch

    parts = [_scene("quad_slicer", 257), _scene("quad_slicer", 513)]
    b = cb.DeviceBatch(parts)
    b.step(2)
    first, second = (b.batch.slice(s) for s in (0, 1))
    before = b.cut_masks()
    assert before[first].any() and before[second][::2].any()
    geom = b.sh["geom_idx"][b.batch.merged.shapes.shape_ids[b.batch.shape_offset[0]]]
    b.sh["geom_type"][geom] = scenes.GEOM_PLANE
    b.mask[second.start:second.stop:2] = 0
    torch.cuda.synchronize()
    b.step(3)
    masks = b.cut_masks()
    assert not masks[first].any() and not masks[second][::2].any() and masks[second][1::2].any()
