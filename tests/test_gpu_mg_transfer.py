"""GPU: the multigrid transfers on both sides of the size at which a thread takes a node
instead of one of its components, nested, tabulated and not coarsened along an axis."""
import numpy as np
import pytest

from test_gpu_mg import _penny_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(86, 86, 84), (85, 88, 86), (129, 89, 8)])
def test_mg_transfers(cuda, shape, precision):
    """86 x 86 x 84 (tables on every axis; the first coarse level, 44 x 44 x 43, is above the
    size too), 85 x 88 x 86 (one axis nested), 129 x 89 x 8 (two nested, one not coarsened): the
    Jacobi solution to the tolerance of the other grids' test, in a fifth of its iterations."""
    res = {}
    for pc in ("jacobi", "mg"):
        ctx = _penny_ctx(shape)
        rc, st = ctx.step_u(dict(pc=pc, precision=precision if pc == "mg" else "fp64"))
        assert rc == 0 and st["reason"] > 0, (pc, st)
        res[pc] = (ctx.get_field("U"), st["ksp_its"])
        ctx.close()
    (uj, kj), (um, km) = res["jacobi"], res["mg"]
    assert np.linalg.norm(um - uj) <= 1e-6 * np.linalg.norm(uj)
    assert km * 5 <= kj, (km, kj)
