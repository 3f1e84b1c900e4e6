"""Rounding of the U operator's stencil: no more of it than the element form's on the same inputs.

The element form runs on the same grid when the modulus is given per cell (all cells alike).
Both are compared with the operator as sums of tensor products of 1-D mass, stiffness and
derivative operators in a wider type (FP64 for FP32 applies, extended precision for FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E, NU = 1e10, 0.25  # E exact in FP32 too: the per-cell modulus is stored so


def _along(f, axis, h, kind):
    """The 1-D operator of linear elements: mass M, stiffness K, C = int phi f', D = int phi' f."""
    f = np.moveaxis(f, axis, -1)
    out = np.zeros_like(f)
    d = f[..., 1:] - f[..., :-1]
    lo, hi = {"M": lambda: (h * (f[..., :-1] / 2 + d / 6), h * (f[..., 1:] / 2 - d / 6)),
              "K": lambda: (-d / h, d / h), "C": lambda: (d / 2, d / 2),
              "D": lambda: (-(f[..., 1:] + f[..., :-1]) / 2, (f[..., 1:] + f[..., :-1]) / 2)}[kind]()
    out[..., :-1] += lo
    out[..., 1:] += hi
    return np.moveaxis(out, -1, axis)


def _operator(u, h, lam, mu):
    def term(f, kinds):
        for q in range(3):
            f = _along(f, 2 - q, h[q], kinds[q])
        return f
    y = [0, 0, 0]
    for c in range(3):
        for d in range(3):
            k = ["M"] * 3
            k[d] = "K"
            y[c] = y[c] + (lam + 2 * mu if d == c else mu) * term(u[..., c], k)
            if d == c:
                continue
            k = ["M"] * 3
            k[c], k[d] = "D", "C"
            y[c] = y[c] + lam * term(u[..., d], k)
            k[c], k[d] = "C", "D"
            y[c] = y[c] + mu * term(u[..., d], k)
    return np.stack(y, -1)


def _fields(n, h):
    Z, Y, X = np.meshgrid(*(np.arange(k) * s for k, s in zip(n[::-1], h[::-1])), indexing="ij")
    smooth = np.stack([np.sin(1.3 * X + .2) * np.cos(.9 * Y + .3 * Z), np.cos(1.1 * X - .4 * Y) * np.sin(.8 * Z + .1),
                       np.sin(.7 * X + .6 * Y + .9 * Z)], -1)
    fine = np.stack([np.sin(13 * X + .2) * np.cos(9 * Y + 3 * Z), np.cos(11 * X - 4 * Y) * np.sin(8 * Z + .1),
                     np.sin(7 * X + 6 * Y + 9 * Z)], -1)
    return dict(random=np.random.default_rng(3).standard_normal(smooth.shape), smooth=smooth, fine=fine,
                moved=smooth + 10)


@pytest.mark.parametrize("prec,n,l,v", [
    ("mixed", (129, 129, 129), (4.0, 4.0, 4.0), 1.0), ("mixed", (129, 121, 113), (4.0, 3.1, 2.2), 0.6),
    ("fp64", (86, 87, 88), (4.0, 4.0 * 86 / 85, 4.0 * 87 / 85), 1.0), ("fp64", (86, 87, 88), (4.0, 3.1, 2.2), 0.6)])
def test_no_more_rounding_than_the_element_form(cuda, prec, n, l, v):
    import torch
    import vpfhf_b200 as vg
    code = vg.MIXED if prec == "mixed" else vg.FP64
    T, R = (np.float32, np.float64) if prec == "mixed" else (np.float64, np.longdouble)
    eta = 1e-8
    ctx = vg.VFContext(n, l, dict(E=E, nu=NU, Gc=100.0), epsilon=0.1, eta=eta, atnum=1)
    ctx.set_bc(vg.rollers())
    ctx.set_field("V", np.full(ctx.N, v))
    ctx.time_step_prepare()
    free = np.ones(n[::-1] + (3,), bool)  # rollers: the other rows are y = x
    free[:, :, [0, -1], 0] = free[:, [0, -1], :, 1] = free[[0, -1], :, :, 2] = False
    h = [R(a) / (k - 1) for a, k in zip(l, n)]
    lam, mu = R(E) * R(NU) / ((1 + R(NU)) * (1 - 2 * R(NU))), R(E) / (2 * (1 + R(NU)))
    # the rows inside the box and those on its faces and edges apart: other code writes them
    inner = np.zeros(n[::-1], bool)
    inner[1:-1, 1:-1, 1:-1] = True
    parts = [free & inner[..., None], free & ~inner[..., None]]
    xs = {name: (u * 1e-4).astype(T) for name, u in _fields(n, [float(a) for a in h]).items()}
    refs = {name: _operator(u.astype(R), h, lam, mu) * (R(T(v)) ** 2 + R(eta)) for name, u in xs.items()}
    err = {}
    for form, modulus in (("stencil", None), ("element", np.full(np.prod([k - 1 for k in n]), E))):
        ctx.set_cell_modulus(modulus)
        for name, u in xs.items():
            x = torch.from_numpy(u.reshape(-1)).cuda()
            y = torch.empty_like(x)
            ctx.u_apply_dev(x, y, code)
            torch.cuda.synchronize()
            ref = refs[name]
            d = y.cpu().numpy().reshape(ref.shape).astype(R) - ref
            err[form, name] = [float(np.sqrt((d[p] ** 2).sum() / (ref[p] ** 2).sum())) for p in parts]
    ctx.close()
    for name in xs:
        for s, e in zip(err["stencil", name], err["element", name]):
            assert s <= e, err


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_values_that_are_not_finite_stay_with_their_neighbours(cuda, prec):
    """A row takes the node's 27 neighbours and nothing else."""
    import torch
    import vpfhf_b200 as vg
    n = (129, 97, 129)  # 4 x 12 tiles x 129 planes: both precisions take the stencil
    ctx = vg.VFContext(n, (4.0,) * 3, dict(E=E, nu=NU, Gc=100.0), epsilon=0.1, eta=1e-8, atnum=1)
    ctx.set_bc(vg.rollers())
    ctx.set_field("V", np.ones(ctx.N))
    ctx.time_step_prepare()
    code, T = (vg.FP64, torch.float64) if prec == "fp64" else (vg.MIXED, torch.float32)
    at = [(40, 33, 65), (1, 50, 64), (127, 16, 1), (64, 0, 70), (0, 31, 20), (128, 96, 128), (50, 0, 128)]
    x = torch.randn(3 * ctx.N, device="cuda", dtype=T, generator=torch.Generator("cuda").manual_seed(1))
    near = np.zeros(n[::-1], bool)
    g = x.view(n[2], n[1], n[0], 3)
    for q, (i, j, k) in enumerate(at):
        g[k, j, i, q % 3] = float("inf") if q & 1 else float("nan")
        near[max(k - 1, 0):k + 2, max(j - 1, 0):j + 2, max(i - 1, 0):i + 2] = True
    y = torch.empty_like(x)
    ctx.u_apply_dev(x, y, code)
    torch.cuda.synchronize()
    fin = np.isfinite(y.cpu().numpy().reshape(n[::-1] + (3,)))
    ctx.close()
    assert fin[~near].all()
    for i, j, k in at:  # (Dirichlet rows are y = x)
        assert not fin[k, j, i].all()
