"""Every instantiation of the persistent FP32 PCG that the dispatch can reach, and
the separate kernels in pairs, drive the mixed solve through the same FP32
iterations.

The FP64 residual repairs a wrong FP32 product or sum at the price of more
iterations, so iterations and refinement rounds are compared as well as x.  The
two sides' dots are grouped differently but agree to some 2^-50, and scalars are
rounded to FP32 before use: counts are equal unless such a rounding falls on the
middle (some 10^-8 of the scalars), which moves a count by a few; 1 % allows for
that.  x agrees to the refinement target (1e-10 of the load) times the
conditioning, taken as 100.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def trials(dims, k, tmp, **env):
    out = str(tmp / "t.npz")
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import numpy as np, specfem3d_geotech_gb300 as sg
        from specfem3d_geotech_gb300 import meshgen
        model = sg.Model(meshgen.slope3d(*%r), precision=sg.PREC_MIXED)
        model.ctx.profile(True)
        r, x = model.trials([1.0 + 0.02 * t for t in range(%d)], sg.make_control(nl_maxiter=1, precision=sg.PREC_MIXED),
                            want_x=True)
        names = ("cg_tot", "nl_iter", "refine_steps", "errcode")
        np.savez(%r, x=x, one_kernel=model.ctx.profile_read()["persistent_ms"] > 0,
                 **{n: [t[n] for t in r] for n in names})
    """ % (ROOT, dims, k, out)
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, env=dict(os.environ, **env))
    return {k: v for k, v in np.load(out).items()}


def same(a, b):
    assert not a["errcode"].any() and not b["errcode"].any()
    assert np.array_equal(a["nl_iter"], b["nl_iter"]) and np.array_equal(a["refine_steps"], b["refine_steps"])
    assert np.all(np.abs(a["cg_tot"] - b["cg_tot"]) <= 0.01 * b["cg_tot"]), (a["cg_tot"], b["cg_tot"])
    for x, y in zip(a["x"], b["x"]):
        assert np.linalg.norm(x - y) <= 1e-8 * np.linalg.norm(y)


# elements: pieces a thread holds (0 to 4 streamed, more streamed) by columns
@pytest.mark.parametrize("dims, k", [
    ((2, 2, 2), 1), ((2, 2, 2), 2), ((2, 2, 2), 16),        # fewer pieces than a block's threads: 1 each
    ((13, 7, 9), 1), ((13, 7, 9), 5), ((13, 7, 9), 16),     # 819: 1, 1, 2
    ((29, 11, 13), 1), ((29, 11, 13), 3), ((29, 11, 13), 8),   # 4,147: 2, 2, streamed
    ((30, 18, 17), 1), ((30, 18, 17), 2), ((30, 18, 17), 4),   # 9,180: 4, 4, streamed
    ((40, 22, 21), 1), ((40, 22, 21), 2),                   # 18,480: 8, streamed
    ((50, 30, 27), 1),                                      # 40,500: streamed
    ((29, 11, 13), 2), ((13, 7, 9), 4), ((34, 20, 20), 4),  # 2, 1, streamed, more than four
    ((19, 9, 11), 8), ((19, 9, 13), 16),                    # 1,881: 2; 2,223: streamed
    ((20, 11, 13), 11), ((26, 16, 16), 7)])                 # 2,860, 6,656: streamed, more than four
def test_persistent_forms_iterate_like_the_separate_kernels(tmp_path, dims, k):
    a = trials(dims, k, tmp_path, SG_PERSIST="1")
    b = trials(dims, k, tmp_path, SG_PERSIST="0")
    assert a["one_kernel"] and not b["one_kernel"]
    same(a, b)


@pytest.mark.parametrize("k", [1, 2, 3, 8, 16])
@pytest.mark.parametrize("dims", [(2, 2, 2), (11, 5, 3), (37, 21, 20)])
def test_flat_kernels_iterate_like_the_staged_gather(tmp_path, dims, k):
    """Up to 15,540 elements: one node a thread of the gather, and several."""
    same(trials(dims, k, tmp_path, SG_PERSIST="0", SG_GATHER_VARIANT="1"),
         trials(dims, k, tmp_path, SG_PERSIST="0", SG_GATHER_VARIANT="0"))


@pytest.mark.parametrize("k", [1, 2, 3, 8, 16])
@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 1, 11), (13, 7, 9)])
def test_matrix_free_applies_iterate_like_stored_matrices(tmp_path, dims, k):
    """Another operator, rounded otherwise: about as many iterations, and the
    same solution."""
    a = trials(dims, k, tmp_path, SG_PERSIST="0", SG_APPLY_VARIANT="5")
    b = trials(dims, k, tmp_path, SG_PERSIST="0", SG_APPLY_VARIANT="1")
    for x, y in zip(a["x"], b["x"]):
        assert np.linalg.norm(x - y) <= 1e-8 * np.linalg.norm(y)
    assert np.all(np.abs(a["cg_tot"] - b["cg_tot"]) <= 0.1 * b["cg_tot"]), (a["cg_tot"], b["cg_tot"])
