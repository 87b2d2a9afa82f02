"""Contexts of one process: what one of them chooses must not break another."""
import os

import numpy as np
import pytest

import specfem3d_geotech_gb300 as sg
from specfem3d_geotech_gb300 import meshgen

pytestmark = pytest.mark.gpu


def test_a_model_outlives_another_choice_of_the_fp32_operator(monkeypatch):
    """SG_APPLY_VARIANT is read by each new context and holds for the process;
    a mixed model built before keeps an operator that it has."""
    ctl = sg.make_control(nl_maxiter=2, precision=sg.PREC_MIXED)
    mesh = meshgen.slope3d(9, 4, 5)
    first = os.environ.get("SG_APPLY_VARIANT", "5")
    a = sg.Context(0)
    model = sg.Model(mesh, precision=sg.PREC_MIXED, ctx=a)
    _, x = model.trials([1.0, 1.1, 1.2], ctl, want_x=True)
    try:
        for variant in ("1", "3", "2"):
            monkeypatch.setenv("SG_APPLY_VARIANT", variant)
            b = sg.Context(0)
            _, y = model.trials([1.0, 1.1, 1.2], ctl, want_x=True)
            assert np.array_equal(x, y)        # the same operator as before
            own = sg.Model(mesh, precision=sg.PREC_MIXED, ctx=b)
            _, z = own.trials([1.0, 1.1, 1.2], ctl, want_x=True)
            # another operator: equal to the refinement target times the conditioning
            assert np.linalg.norm(z - x) <= 1e-8 * np.linalg.norm(x)
            own.close()
            b.close()
    finally:
        monkeypatch.setenv("SG_APPLY_VARIANT", first)
        sg.Context(0).close()
