"""The profile of a solve whose PCG runs inside one kernel: the total stays the
total, and bench.py does not take the FP64 residual's applies for it."""
import pytest

import bench

PROF = dict(total_ms=0.0, apply_ms=6.0, gather_ms=3.0, update_ms=0.5, stress_ms=2.0, stiffness_ms=0.0, persistent_ms=0.0,
            apply_launches=3, launches=100, pcg_iters=400, refine_residuals=3)


def test_report_of_separate_kernels():
    roof, ms = bench.kernel_report(PROF, 192000, 4633520, 8, 2)
    assert roof["kernel"] == "k_apply_mf_planes<8>" and roof["avg_launch_ms"] == 2.0
    assert roof["algorithmic_bytes_per_launch"] == 192000 * 27 * 52 + 2 * 4633521 * 32
    assert ms == {"apply": 2.0, "gather": 1.0, "update": 0.5 / 3, "stress_per_step": 1.0}


def test_report_of_the_persistent_kernel():
    roof, ms = bench.kernel_report(dict(PROF, persistent_ms=20.0), 576, 16000, 8, 2)
    assert roof["kernel"] == "k_pcg_persistent<8>" and roof["avg_iteration_ms"] == 0.05
    assert "avg_launch_ms" not in roof and ms == {"persistent": 0.05, "stress_per_step": 1.0}


@pytest.mark.gpu
@pytest.mark.parametrize("prec, k", [("PREC_MIXED", 8), ("PREC_FP64", 1), ("PREC_FP64", 2)])
def test_total_is_the_sum(built_lib, prec, k):
    import specfem3d_geotech_gb300 as sg
    from specfem3d_geotech_gb300 import meshgen

    prec = getattr(sg, prec)
    model = sg.Model(meshgen.slope3d(9, 4, 5), precision=prec, ctx=sg.Context(0))
    model.ctx.profile(True)
    model.trials([1.0 + 0.02 * t for t in range(k)], sg.make_control(nl_maxiter=2, precision=prec))
    p = model.ctx.profile_read()
    one_kernel = prec == sg.PREC_MIXED or k == 1
    assert (p["persistent_ms"] > 0) == one_kernel and p["apply_ms"] > 0 and p["pcg_iters"] > 0
    parts = ("apply_ms", "gather_ms", "update_ms", "stress_ms", "stiffness_ms", "persistent_ms")
    assert p["total_ms"] == pytest.approx(sum(p[n] for n in parts), rel=1e-12)
