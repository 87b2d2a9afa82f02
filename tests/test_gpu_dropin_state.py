"""What a context keeps between calls of the drop-in must not change what a
later call is refused or allowed."""
import os
import subprocess
import sys

import numpy as np
import pytest

import specfem3d_geotech_gb300 as sg

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def apart(n, seed=3):
    """n unconnected elements with diagonal matrices, and the solution."""
    rng = np.random.default_rng(seed)
    d, f = rng.uniform(1.0, 2.0, 81 * n), rng.standard_normal(81 * n)
    k = np.zeros((n, 81, 81))
    k[:, np.arange(81), np.arange(81)] = d.reshape(n, 81)
    ge = (1 + np.arange(81 * n, dtype=np.int32)).reshape(n, 81)
    return 81 * n, k, np.r_[0.0, f], np.r_[0.0, np.ones(81 * n)], ge, np.r_[0.0, f / d]


def solve(ctx, n):
    neq, k, f, dinv, ge, exact = apart(n)
    u = np.zeros(neq + 1)
    _, err, _ = sg.pcg_solver(neq, n, k, u, f, dinv, ge, 500, 1e-12, ctx=ctx)
    assert err == sg.SG_OK and np.allclose(u, exact, rtol=1e-9, atol=1e-9)


def test_map_of_a_refused_call_is_checked_again():
    """A call whose topology does not fit leaves no trusted map behind: with
    fewer equations, the same map is out of range."""
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import numpy as np, specfem3d_geotech_gb300 as sg
        from tests.test_gpu_dropin_state import apart
        n = 50
        neq, k, f, dinv, ge, _ = apart(n)
        one = np.tile(ge[0], (n, 1))           # all elements on one element's dofs
        few = (81, n, k, np.zeros(82), f[:82], dinv[:82])
        def used(budget):
            ctx = sg.Context(0, budget)
            assert sg.pcg_solver(*few, one, 500, 1e-10, ctx=ctx)[1] == 0
            return ctx
        ctx = used(used(0).hbm_used + 10000)   # the second map's topology takes 21 kB more
        codes = []
        for args in ((neq, n, k, np.zeros(neq + 1), f, dinv), few):
            try:
                sg.pcg_solver(*args, ge, 500, 1e-10, ctx=ctx)
            except sg.SgError as e:
                codes.append(e.code)
        assert codes == [sg.SG_ERR_OOM, sg.SG_ERR_BADARG], codes
        assert sg.pcg_solver(*few, one, 500, 1e-10, ctx=ctx)[1] == 0
    """ % ROOT
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, timeout=300, env=dict(os.environ, SG_PERSIST="0"))


def rows_bytes(n):
    return 4618 * 8 * n   # the packed matrices a solve of n elements may keep


def needs(n):
    """Device bytes of a context after one solve, without the packed rows."""
    ctx = sg.Context(0)
    solve(ctx, n)
    return ctx.hbm_used - rows_bytes(n)


def test_a_larger_solve_fits_after_a_smaller_one():
    ctx = sg.Context(0, needs(400) + 65536)
    solve(ctx, 100)
    kept = ctx.hbm_used
    assert kept > rows_bytes(100) + needs(100) - 65536   # the first solve's rows were kept
    solve(ctx, 400)
    solve(ctx, 100)


def test_a_model_fits_after_a_solve():
    from specfem3d_geotech_gb300 import meshgen

    mesh = meshgen.slope3d(6, 5, 5)
    ctx = sg.Context(0)
    before = ctx.hbm_used
    model = sg.Model(mesh, ctx=ctx)
    room = ctx.hbm_used - before
    model.close()
    n = 20
    assert rows_bytes(n) < room / 4
    ctx = sg.Context(0, needs(n) + room + 65536)
    solve(ctx, n)
    assert ctx.hbm_used >= needs(n) + rows_bytes(n)
    sg.Model(mesh, ctx=ctx).close()
    solve(ctx, n)


def test_a_solve_whose_vectors_do_not_fit_is_refused():
    """Budgets that end anywhere among the solve's buffers: refused, not run
    with a missing one, and the context stays usable."""
    n = 40
    neq, k, f, dinv, ge, _ = apart(n)
    full = needs(n)
    for short in range(1, 40):
        ctx = sg.Context(0, full - short * 8 * (neq + 1) // 4)
        with pytest.raises(sg.SgError) as e:
            sg.pcg_solver(neq, n, k, np.zeros(neq + 1), f, dinv, ge, 500, 1e-12, ctx=ctx)
        assert e.value.code == sg.SG_ERR_OOM
        solve(ctx, 2)
        ctx.close()
