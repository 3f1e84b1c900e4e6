"""GPU: the device-side CG loops -- iteration caps and time limits that end them anywhere in
their body, systems of a few unknowns, and many solves side by side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(n=(9, 8, 7), atnum=1):
    import vpfhf_b200 as vg
    ctx = vg.VFContext(n, (1.0, 1.0, 1.0), dict(E=1e10, nu=0.25, Gc=100.0), epsilon=0.25, eta=1e-8,
                       atnum=atnum, pressurize=True)
    ctx.set_bc(vg.rollers())
    ctx.set_field("pressure", np.full(ctx.N, 1e6))
    ctx.init_cracks([dict(center=(0.5, 0.5, 0.5), r=0.2, theta=0.0, phi=0.0, thickness=0.1)])
    ctx.time_step_prepare()
    return ctx


@pytest.mark.parametrize("maxit", [1, 2, 3, 4, 5, 8, 11])
def test_iteration_cap(cuda, maxit):
    """ksp_maxit its per linear solve: exactly that many, whatever the loop's body holds; the
    capped solves approach the full one."""
    ctx = _ctx()
    rc, st = ctx.step_u(dict(ksp_maxit=maxit, snes_maxit=1))
    assert st["ksp_its"] == maxit and st["newton_its"] == 1
    u1 = ctx.get_field("U")
    ctx.close()
    ctx = _ctx()
    ctx.step_u(dict(ksp_maxit=maxit, snes_maxit=1))
    assert np.array_equal(ctx.get_field("U"), u1)
    ctx.close()


@pytest.mark.parametrize("precision,n", [("fp64", (3, 3, 3)), ("mixed", (3, 4, 3)), ("fp64", (9, 8, 7))])
def test_time_limit_does_not_change_a_solve(cuda, precision, n):
    """With a limit the loop returns to the host every 64 iterations: a solve that ends in time
    takes the same iterations to the same bits as one without."""
    res = []
    for limit in (0.0, 300.0):
        ctx = _ctx(n)
        rc, st = ctx.step_u(dict(precision=precision, time_limit=limit))
        assert rc == 0, st
        rcv, sv = ctx.step_v(dict(precision=precision, time_limit=limit))
        assert rcv == 0, sv
        res.append((ctx.get_field("U"), ctx.get_field("V"), st["ksp_its"], sv["ksp_its"]))
        ctx.close()
    assert res[0][2:] == res[1][2:]
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1])


def test_solves_side_by_side_keep_their_bits(cuda):
    """Jacobi solves of one problem on four workers at once, beside others: every copy ends with
    the bits it has alone (the loop's kernels share the device block by block)."""
    import dataclasses
    from vpfhf_b200.serve import Server, serving_stream
    base = serving_stream(count=4, seed=5, edges=(33, 49), am_its=2, pc="jacobi")
    alone = {}
    for i, p in enumerate(base):
        with Server(workers=1) as srv:
            srv.submit(p)
            alone[i] = srv.next(300.0)
    with Server(workers=4) as srv:
        for k in range(6):
            for i, p in enumerate(base):
                srv.submit(dataclasses.replace(p, tag=4 * k + i))
        for _ in range(24):
            r = srv.next(300.0)
            a = alone[r["tag"] % 4]
            for key in ("elastic", "pressure_work", "surface", "cov", "am_err", "ksp_its_u", "ksp_its_v"):
                assert r[key] == a[key], (r["tag"], key)


@pytest.mark.parametrize("precision,n", [("fp64", (17, 9, 13)), ("mixed", (17, 9, 13)), ("mixed", (18, 18, 10))])
@pytest.mark.parametrize("maxit", [1, 2, 5])
def test_multigrid_iteration_cap(cuda, precision, n, maxit):
    """The multigrid PCG's loop ends at the cap (odd and even unknown counts) with the last step
    in x: the same bits each time, and a residual that Jacobi CG needs more iterations for."""
    out = []
    for pc in ("mg", "mg", "jacobi"):
        ctx = _ctx(n, 2)
        rc, st = ctx.step_u(dict(pc=pc, precision="fp64" if pc == "jacobi" else precision, ksp_maxit=maxit,
                                 snes_maxit=1, ksp_rtol=1e-14))
        assert st["ksp_its"] == maxit, st
        out.append((ctx.get_field("U"), st["fnorm"]))
        ctx.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1] and np.isfinite(out[0][1])
    if maxit == 5:
        assert out[0][1] < out[2][1]

