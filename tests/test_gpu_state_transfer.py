"""F and C of the solver as rows of 9 (copy_particle_state / set_particle_state): exact values at the
edges of the 256-particle tile, at 4-byte aligned offsets and for fewer particles than the solver
holds; arrays a kernel does not take (odd addresses) and arrays that overlap give the copies'
results."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
from crmpm_b200 import scenes  # noqa: E402


@pytest.fixture(scope="module")
def ds():
    sc = scenes.cube_drop()  # 4096 particles
    return cb.DeviceScene(sc, num_max=4101)


@pytest.mark.parametrize("n", [1, 255, 256, 257, 513, 4096, 4101])
@pytest.mark.parametrize("offset", [0, 4, 12, 2])
def test_rows_round_trip(ds, n, offset):
    import torch

    rng = np.random.default_rng(n + offset)
    all_F, all_C = (rng.normal(size=(4101, 9)).astype(np.float32) for _ in range(2))
    whole = [torch.from_numpy(a).to(ds.device) for a in (all_F, all_C)]
    torch.cuda.synchronize()
    ds.solver.set_particle_state(4101, whole[0].data_ptr(), whole[1].data_ptr())
    part_F, part_C = (rng.normal(size=(n, 9)).astype(np.float32) for _ in range(2))
    raw = [torch.zeros(36 * n + 16, dtype=torch.uint8, device=ds.device) for _ in range(4)]
    for t, a in zip(raw, (part_F, part_C)):
        t[offset:offset + 36 * n] = torch.from_numpy(a.reshape(-1).view(np.uint8)).to(ds.device)
    torch.cuda.synchronize()
    ds.solver.set_particle_state(n, raw[0].data_ptr() + offset, raw[1].data_ptr() + offset)
    ds.solver.copy_particle_state(n, raw[2].data_ptr() + offset, raw[3].data_ptr() + offset)
    back = [torch.empty((4101, 9), device=ds.device) for _ in range(2)]
    ds.solver.copy_particle_state(4101, back[0].data_ptr(), back[1].data_ptr())
    ds.sync()
    for t, a in zip(raw[2:], (part_F, part_C)):
        h = t.cpu().numpy()
        np.testing.assert_array_equal(h[offset:offset + 36 * n].view(np.float32).reshape(n, 9), a)
        assert not h[:offset].any() and not h[offset + 36 * n:].any()
    for t, part, full in zip(back, (part_F, part_C), (all_F, all_C)):
        np.testing.assert_array_equal(t.cpu().numpy(), np.concatenate([part, full[n:]]))


def test_overlapping_outputs_hold_the_later_matrix(ds):
    import torch

    n = 300
    F, C = (torch.randn((n, 9), device=ds.device) for _ in range(2))
    torch.cuda.synchronize()
    ds.solver.set_particle_state(n, F.data_ptr(), C.data_ptr())
    out = torch.empty((n, 9), device=ds.device)
    ds.solver.copy_particle_state(n, out.data_ptr(), out.data_ptr())
    ds.sync()
    assert torch.equal(out, C)
