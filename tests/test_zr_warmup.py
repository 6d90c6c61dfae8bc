"""The start of a segment of the fused z/r filter behind a steep front: the sensor's quantities
are 1e8 times larger on the columns left of F, for every F at which the z recurrence of some
segment could start without them (segments start at multiples of 16 positions). What a segment's
warm-up leaves out of the recurrence's history has to stay below rounding at the points right
of the front, whose values are small beside the front's. ComputeRHS against the CPU oracle.

Tolerance: the bar of the FP64 right-hand side, 1e-12, of the largest value right of the front
(velocities share one scale). The recurrence's dominant root is about 0.47: what a warm-up of 64
positions leaves out is below 1e8 * 0.47**64 = 1e-13 of the values behind the front, one of 48
positions about 1e-8."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures

REL = 1e-12
FRONT = 1e8


@pytest.mark.gpu
@pytest.mark.parametrize("Nz,Nr", [(401, 40), (640, 97), (1801, 61)])
def test_rhs_behind_a_front(oracle_mod, Nz, Nr):
    c = fixtures.make_case(Nz, Nr, 30.0, 15.0, 1.2, 2000.0, sc=True, dt_mode=1)
    rng = np.random.default_rng(7)
    for e in (0, 1, 3, 4):
        c["pv"][e] += 0.01 * rng.standard_normal(c["pv"][e].shape)
    p = axj.patches_from_records(c["records"], Nz, Nr)
    dev = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
    ora = oracle_mod.Oracle(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
    dev.set_state(c["pv"], c["target"])
    ora.set_state(c["pv"], c["target"])
    # (the coefficients act from z = 10 on: a third of the columns)
    fronts = list(range((Nz // 3 + 47) // 16 * 16, Nz - 80, 16))
    for F in fronts[:12] + fronts[12::5]:
        pv = c["pv"].copy()
        pv[0, :, :F] *= FRONT
        a, b = dev.compute_rhs(pv), ora.compute_rhs(pv)
        w = slice(F + 46, F + 80)
        v = max(np.abs(b[k][:, w]).max() for k in (1, 2, 3))
        for k in range(5):
            scale = v if k in (1, 2, 3) else np.abs(b[k][:, w]).max()
            assert np.abs(a[k] - b[k])[:, w].max() <= REL * scale, (F, k)
    dev.close()
