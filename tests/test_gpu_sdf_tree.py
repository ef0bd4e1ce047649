"""The mesh SDF's tree walks at the edges of the tree: triangle counts around a leaf and around a full
level, slivers and repeated triangles, closed meshes of few and many triangles.  Grids equal the CPU
restatement bit for bit (distances, off-mesh pattern, signs, gradients)."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
import oracle_py as op  # noqa: E402
from crmpm_b200 import meshes  # noqa: E402


def _same(P, T, cell, **kw):
    got = cb.build_sdf(P, T, cell, 0.02, **kw).host()
    ref = op.port_sdf(P, T, cell, 0.02, **kw)[3]
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(got[~np.isnan(ref)], ref[~np.isnan(ref)])


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 16, 17, 63, 64, 65, 129, 512, 513])
def test_open_soups(n):
    rng = np.random.default_rng(n)
    at = rng.uniform(-0.15, 0.15, size=(n, 1, 3))
    P = (at + rng.normal(scale=0.03, size=(n, 3, 3))).astype(np.float32)
    if n > 4:
        P[1, 2] = P[1, 0] + 1e-5 * (P[1, 1] - P[1, 0])  # a sliver
        P[3] = P[2]  # the same triangle twice
    T = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    _same(P.reshape(-1, 3), T, 0.02, slicer=True)


@pytest.mark.parametrize("mesh", ["box1", "box3", "sphere0", "sphere2", "torus", "far_box"])
def test_closed_meshes(mesh):
    P, T = {"box1": lambda: meshes.box((0.12, 0.08, 0.1), divisions=1), "box3": lambda: meshes.box((0.12, 0.08, 0.1), divisions=3),
            "sphere0": lambda: meshes.icosphere(0.12, 0), "sphere2": lambda: meshes.icosphere(0.12, 2),
            "torus": lambda: meshes.torus(0.12, 0.04, 24, 12),
            "far_box": lambda: meshes.box((0.05, 0.06, 0.04), center=(0.2, 0.15, -0.1), divisions=4)}[mesh]()
    _same(P, T, 0.0173)
