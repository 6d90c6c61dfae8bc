"""What the points inside a body hold does not reach the flow: a body filled with a large finite
value (as programs mark points without a solution) behaves as one filled with the flow's own
values. In 64 bits the fill squared overflows, in the mixed form the fill squared overflows FP32:
the pressure rho T of a blanked point's neighbours is then infinite, and its derivative at the
point (no stencil row: zero) must stay zero.

Tolerance: none; the flow's points are compared bit for bit."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures


def _run(c, fill):
    pv = c["pv"].copy()
    body = c["ibval"] == 0.0
    if fill is not None:
        for e, v in ((0, fill), (1, 0.0), (2, 0.0), (3, 0.0), (4, fill)):
            pv[e][body] = v
    s = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"],
                         axj.patches_from_records(c["records"], c["Nz"], c["Nr"]))
    s.set_state(pv, c["target"])
    s.run(3)
    out = s.get_state()
    s.close()
    return out, body


@pytest.mark.gpu
@pytest.mark.parametrize("sc", [False, True])
@pytest.mark.parametrize("precision,fill", [(0, 1e200), (1, 1e30)])
def test_large_fill_of_a_body(precision, fill, sc):
    c = fixtures.nozzle_case(Nz=140, Nr=97, iw=31, jb=24, jt=40, sc=sc, precision=precision, dt_mode=1)
    a, body = _run(c, None)
    b, _ = _run(c, fill)
    for e in range(5):
        assert np.array_equal(a[e][~body], b[e][~body]), e
