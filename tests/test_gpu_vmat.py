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
