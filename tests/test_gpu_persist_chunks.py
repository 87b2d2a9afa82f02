"""Solves whose persistent kernel ends before the solve does: the host looks at
the clock between launches, and a solve cut into many launches is the solve."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def trials(dims, k, prec, tmp, **env):
    """Results of k trials in a process of their own, or its error code."""
    out = str(tmp / "t.npz")
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import numpy as np, specfem3d_geotech_gb300 as sg
        from specfem3d_geotech_gb300 import meshgen
        model = sg.Model(meshgen.slope3d(*%r), precision=%d)
        ctl = sg.make_control(nl_maxiter=2, precision=%d)
        try:
            r, x = model.trials([1.0 + 0.02 * t for t in range(%d)], ctl, want_x=True)
            np.savez(%r, x=x, err=0, **{n: [t[n] for t in r] for n in ("cg_tot", "nl_iter", "refine_steps", "errcode")})
        except sg.SgError as e:
            np.savez(%r, err=e.code)
    """ % (ROOT, dims, prec, prec, k, out, out)
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300,
                   env={**os.environ, **{n: str(v) for n, v in env.items()}})
    return np.load(out)


MIXED, FP64 = 1, 0


@pytest.mark.parametrize("prec", [MIXED, FP64])
def test_the_wall_clock_limit_holds_between_launches(tmp_path, prec):
    a = trials((9, 4, 5), 1, prec, tmp_path, SG_PERSIST_CHUNK=7, SG_WALL_LIMIT=0)
    assert a["err"] == -2     # SG_ERR_TIMEOUT


@pytest.mark.parametrize("dims, k, prec", [((2, 2, 2), 1, MIXED), ((9, 4, 5), 3, MIXED), ((13, 7, 9), 8, MIXED),
                                           ((13, 7, 9), 16, MIXED), ((29, 11, 13), 2, MIXED), ((13, 7, 9), 1, FP64),
                                           ((19, 11, 9), 1, FP64)])
def test_a_solve_in_many_launches_is_the_solve_in_one(tmp_path, dims, k, prec):
    """u, r and p cross a launch as they are, and the scalars as FP64: equal in
    FP64, and in FP32 unless an FP64 rounding decides an FP32 one (one in some
    10^8 scalars)."""
    a = trials(dims, k, prec, tmp_path, SG_PERSIST_CHUNK=7)
    b = trials(dims, k, prec, tmp_path)
    assert not a["err"] and not b["err"]
    for key in ("x", "cg_tot", "nl_iter", "refine_steps", "errcode"):
        assert np.array_equal(a[key], b[key]), key
