"""PB-MPM's material constraint at the edges of its fast path: the rotation target of matrices on both
sides of the near-rotation test (singular value spread, mirror images, scales), against the polar
factor in FP64, and steps without solver iterations."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
from crmpm_b200 import scenes  # noqa: E402


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


@pytest.mark.parametrize("scale", [1.0, 1e-3, 3e4])
@pytest.mark.parametrize("spread", [0.0, 1e-6, 0.02, 0.2, 0.24, 0.26, 0.4, 0.7])
def test_rotation_target(spread, scale):
    # singular values 1 +- spread: the fast path ends between 0.24 and 0.26 (two opposite offsets)
    rng = np.random.default_rng(int(spread * 1e6) + 7)
    n = 1024
    U, V = _rotations(rng, n), _rotations(rng, n)
    s = np.stack([np.full(n, 1 + spread), np.full(n, 1.0), np.full(n, 1 - spread)], 1)
    A = (np.einsum("nij,nj,nkj->nik", U, s, V) * scale).astype(np.float32)
    u, _, vt = np.linalg.svd(A.astype(np.float64))
    polar = u @ vt
    R9, used = cb.svd_batch(A.transpose(0, 2, 1).reshape(n, 9))[3:5]
    R = R9.reshape(n, 3, 3).transpose(0, 2, 1)
    # a few roundings of a matrix of condition below 6: 16 units in the last place
    assert np.abs(R - polar.transpose(0, 2, 1)).max() < 16 * 2.0 ** -23 * max(1.0, 1 / (1 - spread))
    assert not used.any()


def test_mirrored_and_degenerate_matrices_take_the_svd():
    A = np.stack([np.diag([1.0, 1.0, -0.9]), np.diag([1.0, 1.0, 0.0]), np.zeros((3, 3))]).astype(np.float32)
    R, used = cb.svd_batch(A.reshape(3, 9))[3:5]
    assert np.isfinite(R).all()
    assert used[0] == 0 and used[1] == 1 and used[2] == 1
    np.testing.assert_allclose(np.linalg.det(R[0].reshape(3, 3).astype(np.float64)), 1.0, atol=1e-6)


def test_no_iterations_only_integrate():
    sc = scenes.pb_cutting(size=(0.08, 0.04, 0.08), iterations=0)
    sc.vel[:, :3] = (0.05, 0.1, -0.02)
    g = cb.DeviceScene(sc)
    g.step(3)
    st = g.state()
    x = sc.pos_mass[:, :3].astype(np.float64)
    v = sc.vel[:, :3].astype(np.float64)
    for _ in range(3):
        x += v * sc.dt
        v += sc.gravity.astype(np.float64) * sc.dt
    np.testing.assert_allclose(st["x"], x, atol=1e-6)
    np.testing.assert_allclose(st["v"], v, atol=1e-6)
    np.testing.assert_array_equal(st["C"], 0)
    # and the solver iterates again afterwards
    g.solver.set_solver_iterations(4)
    g.step(2)
    assert np.isfinite(g.state()["x"]).all() and g.solver.grid_stats()["num_sorted"] == sc.n
