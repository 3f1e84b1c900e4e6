"""GPU: the routes a U apply can take on one grid -- two phases, tiles in one wave or split by
phase field, the fixed-scratch apply, the host-buffer pipeline -- against one another."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(n, rng):
    """Intact, with a random blob across tile seams and a constant block."""
    v = np.ones(n[0] * n[1] * n[2])
    vv = v.reshape(n[2], n[1], n[0])
    a = vv[n[2] // 4: n[2] // 2 + 2, n[1] // 5:, n[0] // 3:]
    a[...] = rng.uniform(0, 1, a.shape)
    vv[: n[2] // 5, : n[1] // 2] = 0.4
    return v


def _noalloc(torch, n, l, v, bits, x, stream=None):
    from vpfhf_b200 import _abi
    L = _abi.lib()
    y = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    rc = L.vfgpu_u_apply_noalloc(C.byref(_abi.Grid(*n, *l)), C.byref(_abi.MatProp(1e10, 0.25, 0.0, 0.0, 1.0)),
                                 1e-8, v.data_ptr(), bits.data_ptr(), x.data_ptr(), y.data_ptr(), stream)
    assert rc == 0, L.vfgpu_last_error().decode()
    torch.cuda.synchronize()
    return y


# one tile; x seams alone; y seams alone; both, ragged; more cells than the fixed scratch holds
# in two phases (58^3, 65^3); one plane
@pytest.mark.parametrize("n", [(33, 9, 40), (66, 9, 20), (20, 40, 13), (37, 21, 13), (66, 40, 35), (58, 58, 58),
                               (65, 65, 65), (97, 25, 2)])
def test_two_phases_and_tiles_have_the_same_bits(cuda, n):
    """The device-buffer apply (two phases on these grids), the fixed-scratch apply (tiles where
    its array does not hold the values of two phases) and the host-buffer pipeline sum every node in the
    tile engine's order: equal bits."""
    import vpfhf_b200 as vg
    torch = cuda
    rng = np.random.default_rng(sum(n))
    stretch = (1.0, 1.0, 1.0) if sum(n) % 2 else (1.0, 1.3, 0.8)  # both forms of the element
    l = tuple(0.125 * (k - 1) * s for k, s in zip(n, stretch))
    ctx = vg.VFContext(n, l, dict(E=1e10, nu=0.25), eta=1e-8)
    ctx.set_bc(vg.rollers())
    N = ctx.N
    bits = np.zeros((n[2], n[1], n[0]), np.uint8)
    bits[:, :, [0, -1]] |= 1
    bits[:, [0, -1], :] |= 2
    bits[[0, -1]] |= 4
    bits = torch.from_numpy(bits.reshape(-1)).cuda()
    x = rng.standard_normal(3 * N) * 1e-3
    xd = torch.from_numpy(x).cuda()
    for v in (_field(n, rng), rng.uniform(0, 1, N)):
        ctx.set_field("V", v)
        y = ctx.u_apply(xd, vg.FP64)
        assert torch.equal(_noalloc(torch, n, l, torch.from_numpy(v).cuda(), bits, xd), y)
        assert np.array_equal(ctx.u_apply(x, vg.FP64), y.cpu().numpy())
    ctx.close()
