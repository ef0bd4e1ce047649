"""A batch of one scene is a batch to the kernels: the flags of its only scene have to reach what the
kernels ask about all scenes, or records and cut masks of a slicer scene are not rebuilt."""
import numpy as np
import pytest

from conftest import cuda_available
from gpu_helpers import rel_pos_err

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
import oracle_py as op  # noqa: E402
from crmpm_b200 import scenes  # noqa: E402


@pytest.mark.parametrize("kind", ["quad_slicer", "mesh_slicer"])
@pytest.mark.parametrize("graph", [True, False])
def test_batch_of_one_scene_matches_the_scene(kind, graph):
    """Six substeps in one call, and in calls of one: the scene in a batch of its own against the FP64
    oracle at the parity bar of the other tests, and against the same scene alone."""
    sc = scenes.contact_scene(kind)
    b, g = cb.DeviceBatch([sc]), cb.DeviceScene(sc)
    b.step(6, graph=graph)
    g.step(6, graph=graph)
    sb, sg = b.state(), g.state()
    o = op.PortOracle(sc, 64)
    o.compute_initial_data()
    o.step(6)
    ref = o.state()
    assert rel_pos_err(sb["x"], ref["x"], sc.pos_mass[:, :3], sc.cell_size) < 1e-4
    np.testing.assert_allclose(sb["v"], ref["v"], atol=1e-3 * np.abs(ref["v"]).max())
    assert rel_pos_err(sb["x"], sg["x"], sc.pos_mass[:, :3], sc.cell_size) < 1e-5
