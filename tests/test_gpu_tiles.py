"""GPU: the assembled V operator and the row-wise energies at the sizes where their tiles can
go wrong (the smallest grids, one node past a block's 31 x 7 node columns, its multiples, a
chunk's last planes), against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (grid, AT1 / AT2, thermal strain, per-cell modulus, layers, NOCOMPRESSION)
CASES = [((2, 2, 2), 1, False, False, False, 0), ((3, 8, 5), 2, True, False, True, 0),
         ((31, 7, 9), 1, False, True, False, 0), ((32, 8, 6), 2, False, False, True, 0),
         ((63, 15, 2), 1, True, False, False, 0), ((33, 9, 10), 2, True, True, False, 1),
         ((62, 14, 17), 1, False, False, True, 1)]


def _setup(oracle_mod, n, atnum, thermal, cellE, layers, unilateral):
    import vpfhf_b200 as vg
    rng = np.random.default_rng(sum(n) + atnum)
    l = tuple(0.1 * (k - 1) * s for k, s in zip(n, (1.0, 1.2, 0.9)))
    nlay, N = (2 if layers else 1), n[0] * n[1] * n[2]
    E, nu, Gc = [1e10, 3e10][:nlay], [0.25, 0.2][:nlay], [100.0, 140.0][:nlay]
    alpha = [1e-5 if thermal else 0.0] * nlay
    lay = np.array([k % 2 for k in range(n[2] - 1)], np.int32) if layers else None
    cE = None
    if cellE:
        cE = (1e10 * np.exp(0.5 * rng.standard_normal((n[0] - 1) * (n[1] - 1) * (n[2] - 1)))).astype(np.float32)
        cE = cE.astype(np.float64)
    kw = dict(epsilon=0.25, eta=1e-6, atnum=atnum)
    o = oracle_mod.Oracle(n, l, E=E if layers else E[0], nu=nu if layers else nu[0],
                          Gc=Gc if layers else Gc[0], alpha=alpha if layers else alpha[0],
                          beta=0.7 if thermal else 0.0, layer=lay, cellE=cE, pressurize=True, unilateral=unilateral, **kw)
    ctx = vg.VFContext(n, l, [dict(E=a, nu=b, Gc=g, alpha=t, beta=0.7 if thermal else 0.0) for a, b, g, t in zip(E, nu, Gc, alpha)],
                       pressurize=True, layer=lay, **kw)
    if cE is not None:
        ctx.set_cell_modulus(cE)
    if unilateral:
        ctx.set_unilateral(1)
    ctx.set_bc(vg.rollers())
    v = np.ones(N)  # intact, a constant block, a random block
    vv = v.reshape(n[2], n[1], n[0])
    vv[: n[2] // 3, : n[1] // 2] = 0.4
    blk = vv[n[2] // 2:, n[1] // 3:, n[0] // 3:]
    blk[...] = rng.uniform(0, 1, blk.shape)
    u, p = rng.standard_normal(3 * N) * 1e-4, rng.uniform(0.5, 1.5, N) * 1e6
    theta = rng.uniform(0, 10, N) if thermal else np.zeros(N)
    for name, f in (("U", u), ("V", v), ("VIrrev", v), ("pressure", p), ("theta", theta)):
        ctx.set_field(name, f)
    return o, ctx, u, v, p, theta


@pytest.mark.parametrize("n,atnum,thermal,cellE,layers,unilateral", CASES)
def test_v_residual_and_energies(cuda, oracle_mod, n, atnum, thermal, cellE, layers, unilateral):
    """Residual entries sum at most 216 Gauss terms of one sign pattern and their rounding is
    ~1e-15 of the largest: 1e-11 of it, as the other residual tests.  The energies are sums of
    rounded terms (1e-13), of which the pressure work and the opening cancel by at most the
    square root of the cells: 1e-10."""
    o, ctx, u, v, p, theta = _setup(oracle_mod, n, atnum, thermal, cellE, layers, unilateral)
    F = ctx.v_residual()
    Fr = o.v_residual_ref(u, v, theta, None, p, v)
    assert np.abs(F - Fr).max() <= 1e-11 * np.abs(Fr).max()
    el_o, pw_o = o.u_energy(u, v, theta, None, p)
    el, _, pw = ctx.u_energy()
    cov, cc = ctx.crack_opening(cell=True)
    cov_o, cc_o = o.cov(u, v, cell=True)
    assert el == pytest.approx(el_o, rel=1e-10) and pw == pytest.approx(pw_o, rel=1e-10)
    assert ctx.v_energy() == pytest.approx(o.v_energy(v), rel=1e-10)
    assert cov == pytest.approx(cov_o, rel=1e-10) and ctx.crack_opening() == cov
    assert np.abs(cc - cc_o).max() <= 1e-10 * np.abs(cc_o).max()
    ctx.close()


@pytest.mark.parametrize("n,atnum,thermal,cellE,layers,unilateral", CASES)
def test_u_load(cuda, oracle_mod, n, atnum, thermal, cellE, layers, unilateral):
    """F_U at U = 0 is minus the load: entries of at most 216 Gauss terms, 1e-11 of the largest as
    above."""
    o, ctx, u, v, p, theta = _setup(oracle_mod, n, atnum, thermal, cellE, layers, unilateral)
    u = np.zeros(3 * o.N)
    ctx.set_field("U", u)
    mask, val = o.bc(oracle_mod.rollers_face())
    F = ctx.u_residual()
    Fr = o.u_residual_ref(u, v, theta, None, p, mask, val)
    assert np.abs(F - Fr).max() <= 1e-11 * np.abs(Fr).max()
    ctx.close()


@pytest.mark.parametrize("case", [CASES[1], CASES[3]])
def test_u_diagonal(cuda, oracle_mod, case):
    """One Jacobi CG iteration from U = 0 moves along z = D^-1 r, D the diagonal of the oracle's
    operator (the step lengths, CG's and Newton's, are the solver's): a handful of roundings of
    sums of one sign, 1e-10."""
    o, ctx, u, v, p, theta = _setup(oracle_mod, *case)
    n3 = 3 * o.N
    ctx.set_field("U", np.zeros(n3))
    mask, val = o.bc(oracle_mod.rollers_face())
    rc, st = ctx.step_u(dict(ksp_maxit=1, snes_maxit=1))
    assert st["ksp_its"] == 1, st
    F = o.u_residual_ref(np.zeros(n3), v, theta, None, p, mask, val)
    D, e = np.empty(n3), np.zeros(n3)
    for i in range(n3):
        e[i] = 1.0
        D[i] = o.u_apply(v, e, mask)[i]
        e[i] = 0.0
    z, U = F / D, ctx.get_field("U")
    i = np.abs(z).argmax()
    assert U[i] / z[i] < 0.0
    assert np.abs(U / U[i] - z / z[i]).max() <= 1e-10
    ctx.close()


# Grids that take the U stencil: the smallest that do in FP64 (2000 units of 32 x 8 x 1), one
# column past a 32 x 16 tile and its multiples, a chunk of few planes, faces not a multiple of
# 30 columns or 4 planes; the last one also in FP32 (6000 units).
STENCIL = [((34, 40, 200), (1.0, 1.0, 5.0)), ((66, 18, 223), (2.0, 0.6, 6.0)), ((35, 129, 64), (34.0, 128.0, 63.0)),
           ((97, 99, 161), (1.1, 0.9, 1.7))]


@pytest.mark.parametrize("n,l", STENCIL)
@pytest.mark.parametrize("field", ["intact", "blob", "scaled"])
def test_u_stencil(cuda, oracle_mod, n, l, field):
    """K(v) x with the stencil at homogeneous nodes, against the oracle (FP64 1e-12 of the
    largest entry, FP32 2e-6 normwise: the bounds of the element operator's tests) and the
    same bits in every split mode; Dirichlet rows on all faces and one vertex, a field that
    is intact, that has a random blob across tile seams and faces, and that is constant at
    0.4 with a blob."""
    import vpfhf_b200 as vg
    E, nu, eta = 1e10, 0.3, 1e-6
    rng = np.random.default_rng(sum(n))
    o = oracle_mod.Oracle(n, l, E=E, nu=nu, eta=eta)
    ctx = vg.VFContext(n, l, dict(E=E, nu=nu), eta=eta)
    bc = vg.rollers()
    bc[0] = vg.BCSpec(X0=vg.BC_ZERO, X1=vg.BC_ZERO, X1Y1Z0=vg.BC_ONE)
    bc[2] = vg.BCSpec(Z0=vg.BC_ZERO, Y1=vg.BC_ZERO)
    ctx.set_bc(bc)
    mask = np.zeros((n[2], n[1], n[0], 3), np.uint8)
    mask[:, :, [0, -1], 0] = 1
    mask[:, [0, -1], :, 1] = 1
    mask[0, :, :, 2] = mask[:, -1, :, 2] = 1
    mask = mask.reshape(-1)
    v = np.full(o.N, 0.4 if field == "scaled" else 1.0)
    if field != "intact":
        vv = v.reshape(n[2], n[1], n[0])
        a = vv[n[2] // 3: n[2] // 3 + 5, 10:21, 25:]
        a[...] = rng.uniform(0, 1, a.shape)
        vv[-2:, :3, :4] = 0.7
    ctx.set_field("V", v)
    x = rng.standard_normal(3 * o.N) * 1e-3
    xd = cuda.from_numpy(x).cuda()
    yref = o.u_apply(v, x, mask)
    y = ctx.u_apply(xd, vg.FP64)
    assert np.abs(y.cpu().numpy() - yref).max() <= 1e-12 * np.abs(yref).max()
    y32 = ctx.u_apply(xd, vg.MIXED)
    assert np.linalg.norm(y32.cpu().numpy() - yref) <= 2e-6 * np.linalg.norm(yref)
    for mode in ("on", "off"):
        ctx.set_u_split(mode)
        assert cuda.equal(ctx.u_apply(xd, vg.FP64), y)
        assert cuda.equal(ctx.u_apply(xd, vg.MIXED), y32)
    # the Dirichlet rows move with the boundary conditions, also when v does not
    ctx.set_bc([vg.BCSpec(), vg.BCSpec(), vg.BCSpec(Z1=vg.BC_ZERO)])
    m2 = np.zeros((n[2], n[1], n[0], 3), np.uint8)
    m2[-1, :, :, 2] = 1
    yref = o.u_apply(v, x, m2.reshape(-1))
    assert np.abs(ctx.u_apply(xd, vg.FP64).cpu().numpy() - yref).max() <= 1e-12 * np.abs(yref).max()
    ctx.close()


@pytest.mark.parametrize("cellE,unilateral,layers", [(False, 1, False), (True, 0, False), (True, 1, False),
                                                     (False, 0, True)])
def test_u_tiles(cuda, oracle_mod, cellE, unilateral, layers):
    """The tile engine past the sizes of the two-phase apply (86 x 87 x 88: more than 400,000
    cells, ragged tiles), where the other forms' tests are on smaller grids: NOCOMPRESSION,
    per-cell modulus, material layers; FP64 at 1e-12, FP32 at 2e-6 against the oracle."""
    import vpfhf_b200 as vg
    n, l = (86, 87, 88), (1.7, 1.6, 1.9)
    rng = np.random.default_rng(21)
    cE = None
    if cellE:
        cE = np.exp(np.log(1e10) + 0.5 * rng.standard_normal((n[0] - 1) * (n[1] - 1) * (n[2] - 1)))
        cE = cE.astype(np.float32).astype(np.float64)
    E, nu = ([1e10, 3e10], [0.25, 0.3]) if layers else ([1e10], [0.25])
    lay = np.array([k // 40 % 2 for k in range(n[2] - 1)], np.int32) if layers else None
    o = oracle_mod.Oracle(n, l, E=E, nu=nu, eta=1e-6, cellE=cE, unilateral=unilateral, layer=lay)
    ctx = vg.VFContext(n, l, [dict(E=a, nu=b) for a, b in zip(E, nu)], eta=1e-6, layer=lay)
    if cE is not None:
        ctx.set_cell_modulus(cE)
    ctx.set_bc(vg.rollers())
    mask, _ = o.bc(oracle_mod.rollers_face())
    v = np.ones(o.N)
    vv = v.reshape(n[2], n[1], n[0])
    vv[30:50, 20:60, 10:70] = rng.uniform(0, 1, (20, 40, 60))
    u0 = rng.standard_normal(3 * o.N) * 1e-4
    ctx.set_field("V", v)
    if unilateral:
        ctx.set_unilateral(1)
        ctx.set_field("U", u0)
    x = rng.standard_normal(3 * o.N) * 1e-3
    yref = o.u_apply_u(u0, v, x, mask) if unilateral else o.u_apply(v, x, mask)
    xd = cuda.from_numpy(x).cuda()
    assert np.abs(ctx.u_apply(xd, vg.FP64).cpu().numpy() - yref).max() <= 1e-12 * np.abs(yref).max()
    y32 = ctx.u_apply(xd, vg.MIXED).cpu().numpy()
    assert np.linalg.norm(y32 - yref) <= 2e-6 * np.linalg.norm(yref)
    ctx.close()
