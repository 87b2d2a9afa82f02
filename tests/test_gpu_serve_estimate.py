"""A request's footprint estimate covers what it uses, and counts FP32 element
matrices only where the operator reads them."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NE, FP32_MATRIX = 30 * 20 * 20, 2432 * 4


def request(variant):
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import specfem3d_geotech_gb300 as sg
        from specfem3d_geotech_gb300 import meshgen
        srv = sg.Server(0, 0, workers=1)
        ctl = sg.make_control(nl_maxiter=3, precision=sg.PREC_MIXED)
        r = srv.wait(srv.submit(meshgen.slope3d(30, 20, 20), ctl, lo=1.0, hi=2.0, step=0.5, k=8), timeout=250)
        print(r["status"], int(r["hbm_bytes"]), int(r["footprint"]))
        srv.close()
    """ % ROOT
    out = subprocess.run([sys.executable, "-c", code], check=True, capture_output=True, text=True, timeout=300,
                         env=dict(os.environ, SG_APPLY_VARIANT=variant)).stdout
    status, used, estimate = (int(v) for v in out.split())
    assert status == 0 and used <= estimate
    return used, estimate


def test_estimate_follows_the_operator():
    free, stored = request("5"), request("3")
    assert stored[0] - free[0] == NE * FP32_MATRIX
    assert abs(stored[1] - free[1] - 1.125 * NE * FP32_MATRIX) <= 2    # an eighth on top of everything
