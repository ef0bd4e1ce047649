"""PB-MPM's rotation target around the edge of Newton's iteration: the squared Frobenius distance 0.25 of
X^T X from the identity at mean square singular value 1, which two opposite offsets reach at a spread
near 0.18, a single one near 0.33 or -0.30 and two equal ones near 0.43 (the widest spectra inside it have
a ratio of 1.46).  On both sides of it the target is the polar factor in FP64 to a few roundings, and no
matrix asks for the FP64 redo."""
import numpy as np
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
from test_gpu_pb_constraint import _rotations  # noqa: E402

SPECTRA = {"opposite": lambda s: (1 + s, 1.0, 1 - s), "one_up": lambda s: (1 + s, 1.0, 1.0), "one_down": lambda s: (1 - s, 1.0, 1.0),
           "two_up": lambda s: (1 + s, 1 + s, 1.0)}
# spreads on both sides of the edge of each
SPREADS = {"opposite": (0.1, 0.15, 0.17, 0.175, 0.18, 0.185, 0.2), "one_up": (0.2, 0.28, 0.31, 0.325, 0.335, 0.35, 0.4),
           "one_down": (0.2, 0.25, 0.28, 0.295, 0.303, 0.32, 0.35), "two_up": (0.25, 0.35, 0.4, 0.42, 0.435, 0.45, 0.5)}


def _beyond(A):
    """How far each matrix is beyond the edge of the fast path, by its criterion in FP64."""
    X = A / np.sqrt((A ** 2).sum(axis=(1, 2), keepdims=True) / 3)
    g = np.einsum("nki,nkj->nij", X, X) - np.eye(3)
    return (g ** 2).sum(axis=(1, 2)) - 0.25


@pytest.mark.parametrize("scale", [1.0, 1e-3, 3e4])
@pytest.mark.parametrize("kind", sorted(SPECTRA))
def test_rotation_target_around_the_edge(kind, scale):
    rng = np.random.default_rng(17)
    n = 512
    beyond = []
    for spread in SPREADS[kind]:
        U, V = _rotations(rng, n), _rotations(rng, n)
        s = np.array(SPECTRA[kind](spread))
        A = (np.einsum("nij,j,nkj->nik", U, s, V) * scale).astype(np.float32)
        A64 = A.astype(np.float64) / scale
        beyond += list(_beyond(A64))
        u, _, vt = np.linalg.svd(A64)
        R9, used = cb.svd_batch(A.transpose(0, 2, 1).reshape(n, 9))[3:5]
        R = R9.reshape(n, 3, 3).transpose(0, 2, 1).astype(np.float64)
        # a few roundings: 16 units in the last place, times the condition
        assert np.abs(R - (u @ vt).transpose(0, 2, 1)).max() < 16 * 2.0 ** -23 * s.max() / s.min()
        assert not used.any()
    beyond = np.array(beyond)
    assert (beyond < -0.05).any() and ((-0.05 < beyond) & (beyond < 0)).any()
    assert ((0 < beyond) & (beyond < 0.05)).any() and (beyond > 0.05).any()
