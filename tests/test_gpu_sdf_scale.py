"""Signs and distances of mesh SDFs far from unit scale: the same closed meshes scaled by powers of two
over the range in which products of three lengths are representable.  Power-of-two scaling of the
mesh, the cell and the bounds scales every intermediate of the distance exactly, so the grid is the unit grid's times the
scale; the sign has to be the unit grid's at every node that is not on the surface."""
import ctypes as C

import numpy as np
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
from crmpm_b200 import meshes  # noqa: E402


def _grid(P, T, cell, lower, dims):
    import torch

    d = cb.SdfDescC()
    d.cellSize = cell
    d.fatten = 0.0
    d.lowerBound[:] = [float(v) for v in lower]
    d.boundingSize[:] = [float(cell * n) for n in dims]
    d.sdfDimension[:] = dims
    d.slicerSpineArea = (C.c_float * 4)(float("nan"), 0.0, 0.0, 0.0)
    m, keep = cb._mesh_struct(P, T)
    out = torch.empty((dims[2], dims[1], dims[0], 4), dtype=torch.float32, device="cuda:0")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    cb.check(cb.lib().CrB200SdfCompute(C.byref(d), C.byref(m), C.c_void_p(out.data_ptr()), 1, st), "CrB200SdfCompute")
    del keep
    return out.cpu().numpy()[..., 3]


@pytest.mark.parametrize("exponent", [-28, -26, -20, 0, 18, 20, 22, 24, 27])
@pytest.mark.parametrize("mesh", ["box", "sphere", "torus"])
def test_signs_at_scale(mesh, exponent):
    P, T = {"box": lambda: meshes.box((1.0, 0.8, 0.9), divisions=2), "sphere": lambda: meshes.icosphere(1.0, 2),
            "torus": lambda: meshes.torus(1.0, 0.35, 24, 12)}[mesh]()
    dims, cell, lower = (23, 21, 22), 0.125, np.array([-1.40625, -1.28125, -1.34375])
    s = 2.0 ** exponent
    unit = _grid(P, T, cell, lower, dims)
    got = _grid((P.astype(np.float64) * s).astype(np.float32), T, cell * s, lower * s, dims)
    assert (unit < 0).sum() > 100 and (unit > 0).sum() > 100
    off = np.abs(unit) > 1e-5
    np.testing.assert_array_equal(np.sign(got)[off], np.sign(unit)[off])
    np.testing.assert_allclose(got, unit * s, rtol=1e-5, atol=1e-5 * s)
