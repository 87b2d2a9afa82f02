"""The FP32 PCG kernels by width and mesh size: each pair of ways to run an
iteration drives the mixed solve to the same trials.

The FP64 residual decides when a solve is done, so two FP32 paths that differ
in rounding only agree to the refinement target (1e-10 of the load) times the
conditioning of these small meshes: 1e-8 is two orders above what that gives,
and far below any wrong sum, column or index.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-8
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def trials(dims, k, tmp, **env):
    out = str(tmp / ("_".join(env.values()) + ".npz"))
    code = ("import sys; sys.path.insert(0, %r); import numpy as np; import specfem3d_geotech_gb300 as sg;"
            "from specfem3d_geotech_gb300 import meshgen; m = sg.Model(meshgen.slope3d(*%r), precision=sg.PREC_MIXED);"
            "r, x = m.trials([1.0 + 0.02 * t for t in range(%d)], sg.make_control(nl_maxiter=2, precision=sg.PREC_MIXED),"
            " want_x=True); np.savez(%r, x=x, nl=[t['nl_iter'] for t in r], e=[t['errcode'] for t in r])") % (
        ROOT, dims, k, out)
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, **env), timeout=300)
    return np.load(out)


def same(a, b):
    assert not a["e"].any() and not b["e"].any() and np.array_equal(a["nl"], b["nl"])
    for x, y in zip(a["x"], b["x"]):
        assert np.linalg.norm(x - y) <= TOL * np.linalg.norm(y)


@pytest.mark.parametrize("k", [1, 2, 3, 5, 16])
@pytest.mark.parametrize("dims", [(2, 2, 2), (11, 5, 3)])
def test_flat_gather_and_update_match_staged(tmp_path, dims, k):
    a = trials(dims, k, tmp_path, SG_PERSIST="0", SG_GATHER_VARIANT="1")
    b = trials(dims, k, tmp_path, SG_PERSIST="0", SG_GATHER_VARIANT="0")
    same(a, b)


@pytest.mark.parametrize("k", [1, 2, 3, 8, 16])
@pytest.mark.parametrize("dims", [(2, 2, 2), (13, 7, 9), (29, 11, 13)])
def test_persistent_matches_separate_kernels(tmp_path, dims, k):
    """8 elements (fewer warps than schedulers), 819 and 4,147 (one, two or
    streamed pieces a thread by k; the element cache full and not)."""
    a = trials(dims, k, tmp_path, SG_PERSIST="1")
    b = trials(dims, k, tmp_path, SG_PERSIST="0")
    same(a, b)


def fp64(dims, tmp, persist):
    out = str(tmp / ("fp64_%s.npz" % persist))
    code = ("import sys; sys.path.insert(0, %r); import numpy as np; import specfem3d_geotech_gb300 as sg;"
            "from specfem3d_geotech_gb300 import meshgen; m = sg.Model(meshgen.slope3d(*%r));"
            "r, x = m.trials([1.1], sg.make_control(nl_maxiter=2), want_x=True);"
            "k, d, f = m.stiffness(); d[1:] = 1 / d[1:]; d[0] = 0; ge = m.arrays()['gdof_elmt'];"
            "u = np.zeros(m.neq + 1); it, e, _ = sg.pcg_solver(m.neq, m.nelmt, k, u, f, d, ge, 5000, 1e-10);"
            "k[0, 0, 80] = k[0, 80, 0] = 1e-3 * abs(k[0, 0, 0]); v = np.zeros(m.neq + 1);"
            "jt, g, _ = sg.pcg_solver(m.neq, m.nelmt, k, v, f, d, ge, 5000, 1e-10);"
            "w = np.zeros(m.neq + 1); n = sg.pcg_solver(m.neq, m.nelmt, k, w, f, d, ge, 3, 1e-10);"
            "np.savez(%r, x=x, u=u, v=v, w=w, it=[it, jt, n[0], r[0]['cg_tot']], e=[e, g, n[1]])") % (ROOT, dims, out)
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, SG_PERSIST=persist), timeout=300)
    return np.load(out)


@pytest.mark.parametrize("dims", [(2, 2, 2), (9, 8, 8), (19, 11, 9)])
def test_fp64_persistent_is_bitwise_the_separate_kernels(tmp_path, dims):
    """8 elements, 576 (matrices stay in shared memory) and 1,881 (they stream);
    the model's sparse matrices, the drop-in's dense ones, a solve that runs
    out, and a dense matrix with an entry between uncoupled nodes, which is not
    packed; that entry meets a fixed dof, so the solution is the packed one's."""
    a, b = fp64(dims, tmp_path, "1"), fp64(dims, tmp_path, "0")
    for key in ("x", "u", "v", "w", "it", "e"):
        assert np.array_equal(a[key], b[key]), key
    assert a["e"].tolist() == [0, 0, -1] and np.array_equal(a["u"], a["v"])


@pytest.mark.parametrize("k", [3, 8, 16])
@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 1, 11), (13, 7, 9)])
def test_plane_apply_matches_stored_matrices(tmp_path, dims, k):
    """One element group, a ragged last group, and more groups than one pass."""
    a = trials(dims, k, tmp_path, SG_PERSIST="0", SG_APPLY_VARIANT="5")
    b = trials(dims, k, tmp_path, SG_PERSIST="0", SG_APPLY_VARIANT="1")
    same(a, b)
