"""GPU: the assembled V operator apart from its tiles' sizes (test_gpu_tiles.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(7, 6, 5), (33, 9, 8), (2, 2, 2), (40, 3, 17)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_that_are_not_finite_stay_with_their_neighbours(cuda, n, bad):
    """K_V v at a node reads the nodes of the elements around it and no others: a value that is
    not finite on a face, an edge or inside reaches those nodes of the residual and none across
    the box."""
    import vpfhf_b200 as vg
    rng = np.random.default_rng(sum(n))
    l = tuple(0.1 * (k - 1) for k in n)
    ctx = vg.VFContext(n, l, dict(E=1e10, nu=0.25, Gc=100.0), epsilon=0.2, eta=1e-6, atnum=2, pressurize=True)
    ctx.set_bc(vg.rollers())
    ctx.set_field("U", rng.standard_normal(3 * ctx.N) * 1e-4)
    for at in ((n[0] - 1, n[1] // 2, n[2] // 2), (0, 0, n[2] - 1), (n[0] // 2, n[1] - 1, 0), tuple(k // 2 for k in n)):
        v = rng.uniform(0, 1, (n[2], n[1], n[0]))
        v[at[2], at[1], at[0]] = bad
        ctx.set_field("V", v.reshape(-1))
        F = ctx.v_residual().reshape(n[2], n[1], n[0])
        near = np.zeros(v.shape, bool)
        near[tuple(slice(max(a - 1, 0), a + 2) for a in at[::-1])] = True
        assert np.isfinite(F[~near]).all()
        assert not np.isfinite(F[at[2], at[1], at[0]])
    ctx.close()


def test_smooth_v_keeps_the_accuracy_of_differences(cuda):
    """K_V v for a smooth v without strain (AT1: the stiffness part alone) against extended
    precision.  The rows are differences of neighbours: of the order of sum |a_ij| times the
    largest difference d between a node and its neighbours, not times v itself.  30 roundings
    (27 products, their sum) of 2^-53 of that, and four of the load subtracted from it; plain
    products would leave about 3 roundings of sum |a_ij| max v, a hundred times as much."""
    import vpfhf_b200 as vg
    n, h = (40, 33, 36), 1.0 / 32
    Gc, eps = 100.0, 20.0 / 32
    l = tuple(h * (k - 1) for k in n)
    ctx = vg.VFContext(n, l, dict(E=1e10, nu=0.25, Gc=Gc), epsilon=eps, eta=1e-6, atnum=1)
    ctx.set_bc(vg.rollers())
    Z, Y, X = np.meshgrid(*(np.arange(k) * h for k in n[::-1]), indexing="ij")
    v = 0.7 + 0.2 * np.sin(0.8 * X) * np.cos(0.5 * Y + 0.3 * Z)
    ctx.set_field("V", np.zeros(ctx.N))
    F0 = ctx.v_residual().reshape(v.shape)  # minus the load
    ctx.set_field("V", v.reshape(-1))
    F = ctx.v_residual().reshape(v.shape)
    ctx.close()
    ld = np.longdouble
    aeps, hl = ld(Gc) / (ld(2) / 3) / 2 * ld(eps), ld(h)

    def along(f, axis, mass):
        f = np.moveaxis(f, axis, -1)
        d = f[..., 1:] - f[..., :-1]
        out = np.zeros_like(f)
        if mass:  # h (f_i / 2 + d / 6) from each element
            out[..., :-1] += hl * (f[..., :-1] / 2 + d / 6)
            out[..., 1:] += hl * (f[..., 1:] / 2 - d / 6)
        else:
            out[..., :-1] -= d / hl
            out[..., 1:] += d / hl
        return np.moveaxis(out, -1, axis)
    K = sum(along(along(along(v.astype(ld), 0, q != 0), 1, q != 1), 2, q != 2) for q in range(3))
    err = np.abs(F.astype(ld) - (aeps * K + F0.astype(ld)))
    d = max(np.abs(np.diff(v, axis=a)).max() for a in range(3)) * 3
    suma = float(aeps * hl) * 16 / 3  # of a cube's 27 couplings
    assert err.max() <= 2.0 ** -53 * (30 * suma * d + 4 * np.abs(F0).max())
