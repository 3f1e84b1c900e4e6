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


def _launches(torch, ctx, prec, x, y):
    """Names of the kernels of one u_apply_dev, from a capture of the ctx's stream."""
    from cuda.bindings import driver as d

    def ok(r):
        assert int(r[0]) == 0, r
        return r[1] if len(r) == 2 else r[1:]
    torch.cuda.synchronize()
    ctx.u_apply_dev(x, y, prec)  # lists built
    st = d.CUstream(ctx.stream_handle)
    ok(d.cuStreamBeginCapture(st, d.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL))
    ctx.u_apply_dev(x, y, prec)
    g = ok(d.cuStreamEndCapture(st))
    nodes, n = ok(d.cuGraphGetNodes(g, 16))
    names = []
    for nd in nodes[:n]:
        p = ok(d.cuGraphKernelNodeGetParams(nd))
        names.append(ok(d.cuFuncGetName(p.func) if int(p.func) else d.cuKernelGetName(p.kern)).decode())
    ok((d.cuGraphDestroy(g)[0], None))
    return names


@pytest.mark.parametrize("n,kind", [((37, 21, 13), "one"), ((66, 40, 35), "cells"), ((45, 37, 33), "layers"),
                                    ((86, 87, 88), "cells"), ((86, 87, 88), "layers")])
def test_split_modes_run_what_they_name(cuda, oracle_mod, n, kind):
    """OFF runs one wave of the general kernel and ON the fixed-weight and the general one, on every
    grid that does not take the stencil, whatever AUTO takes there; per-cell modulus, layers and
    one material, both precisions: equal bits, also after v has changed, FP64 at 1e-12 and FP32 at
    2e-6 of the oracle; and a Jacobi U step (its p.w sums run over the partials of each mode's
    waves, in another order) ends at the same U to the solver's tolerance."""
    import vpfhf_b200 as vg
    torch = cuda
    rng = np.random.default_rng(sum(n))
    l = tuple(0.125 * (k - 1) for k in n)
    E, nu, lay, cE = [1e10], [0.25], None, None
    if kind == "layers":
        E, nu = [1e10, 3e10, 6e9], [0.25, 0.3, 0.2]
        lay = np.array([3 * k // (n[2] - 1) for k in range(n[2] - 1)], np.int32)
    if kind == "cells":
        cE = np.exp(np.log(1e10) + 0.5 * rng.standard_normal((n[0] - 1) * (n[1] - 1) * (n[2] - 1)))
        cE = cE.astype(np.float32).astype(np.float64)
    o = oracle_mod.Oracle(n, l, E=E, nu=nu, eta=1e-6, layer=lay, cellE=cE)
    ctx = vg.VFContext(n, l, [dict(E=e, nu=p) for e, p in zip(E, nu)], eta=1e-6, epsilon=0.25, pressurize=True, layer=lay)
    if cE is not None:
        ctx.set_cell_modulus(cE)
    ctx.set_bc(vg.rollers())
    ctx.set_field("pressure", np.full(ctx.N, 1e6))
    mask, _ = o.bc(oracle_mod.rollers_face())
    x = torch.from_numpy(rng.standard_normal(3 * ctx.N) * 1e-3).cuda()
    x32 = x.float()
    xs = {vg.FP64: x, vg.MIXED: x32}
    u, prev = {}, None
    for v in (_field(n, rng), rng.uniform(0.2, 1, ctx.N), _field(n, rng)):
        ctx.set_field("V", v)
        for prec in (vg.FP64, vg.MIXED):
            ys = {}
            for mode in ("auto", "off", "on"):
                ctx.set_u_split(mode)
                y = torch.empty_like(xs[prec])
                names = _launches(torch, ctx, prec, xs[prec], y)
                ctx.torch_stream().synchronize()
                tiles = [k for k in names if "tile_apply_kernel" in k]
                const = [k for k in tiles if "UOpConst" in k or "UOpF2Const" in k]
                if mode != "auto":
                    assert len(tiles) == (2 if mode == "on" else 1) and len(const) == (mode == "on"), names
                ys[mode] = y
            assert torch.equal(ys["on"], ys["off"]) and torch.equal(ys["auto"], ys["off"])
            yref = o.u_apply(v, xs[prec].double().cpu().numpy(), mask)
            y = ys["on"].double().cpu().numpy()
            if prec == vg.FP64:
                assert np.abs(y - yref).max() <= 1e-12 * np.abs(yref).max()
            else:
                assert np.linalg.norm(y - yref) <= 2e-6 * np.linalg.norm(yref)
    for mode in ("off", "on"):
        for pc in ("jacobi", "mg"):
            ctx.set_u_split(mode)
            ctx.set_field("U", np.zeros(3 * ctx.N))
            rc, st = ctx.step_u(dict(pc=pc, ksp_rtol=1e-12))
            assert rc == 0 and st["reason"] > 0, st
            u[mode, pc] = ctx.get_field("U")
    # two solutions whose preconditioned residuals are at most 1e-12 of the first one's, on a system of condition 1e6 at most
    for pc in ("jacobi", "mg"):
        assert np.abs(u["on", pc] - u["off", pc]).max() <= 1e-6 * np.abs(u["off", pc]).max()
    ctx.close()


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


@pytest.mark.parametrize("n", [(33, 9, 60), (9, 8, 300), (2, 2, 2)])
def test_one_tile_noalloc_calls_may_overlap(cuda, n):
    """Grids of one tile use nothing of the fixed scratch: calls on four streams at once, on
    different vectors, each give the bits they give alone."""
    from vpfhf_b200 import _abi
    torch = cuda
    L, N = _abi.lib(), n[0] * n[1] * n[2]
    rng = np.random.default_rng(3)
    l = tuple(0.125 * (k - 1) for k in n)
    v = torch.from_numpy(rng.uniform(0, 1, N)).cuda()
    bits = torch.from_numpy(rng.integers(0, 8, N).astype(np.uint8)).cuda()
    xs = [torch.from_numpy(rng.standard_normal(3 * N)).cuda() for _ in range(4)]
    alone = [_noalloc(torch, n, l, v, bits, x) for x in xs]
    g, mp = _abi.Grid(*n, *l), _abi.MatProp(1e10, 0.25, 0.0, 0.0, 1.0)
    streams = [torch.cuda.Stream() for _ in xs]
    ys = [[torch.full_like(x, float("nan")) for _ in range(50)] for x in xs]
    torch.cuda.synchronize()
    for k in range(50):
        for s, x, y in zip(streams, xs, ys):
            rc = L.vfgpu_u_apply_noalloc(C.byref(g), C.byref(mp), 1e-8, v.data_ptr(), bits.data_ptr(), x.data_ptr(),
                                         y[k].data_ptr(), s.cuda_stream)
            assert rc == 0, L.vfgpu_last_error().decode()
    torch.cuda.synchronize()
    for y, a in zip(ys, alone):
        assert all(torch.equal(q, a) for q in y)
