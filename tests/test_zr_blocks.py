"""The row blocks and segments of the fused z/r filter: ComputeRHS with shock capturing on
grids whose rows end at, before and after the 40 rows of a compact block, whose wall patches put
closure rows (with their 11-point windows) and blanked points anywhere in a block and across
its edges, and whose lengths end inside and at a segment's blocks of 16 positions, against the
CPU oracle.

The solution is perturbed by 1 % at every point, so that the sensor's fourth differences do not
cancel and its coefficients act everywhere (a step of so rough a state can be unstable, its
right-hand side is not). Tolerance: the bar of the FP64 right-hand side, 1e-12 of each field's
largest value (velocities share one scale)."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures
from axisymmetricjet_b200._ffi import NSCBC_NOSLIP_WALL, SAT_NOSLIP_WALL

REL = 1e-12
CASES = [("jet", Nz, Nr) for Nz, Nr in [(12, 12), (15, 39), (16, 40), (17, 41), (47, 45), (48, 79), (64, 80), (65, 81),
                                        (130, 121), (700, 46), (40, 300)]]
CASES += [("nozzle", 90, 97, iw, jb, jt) for iw, jb, jt in [(20, 24, 28), (16, 33, 40), (31, 36, 41), (32, 39, 45),
                                                           (45, 44, 50), (60, 70, 80), (17, 80, 86)]]


def _case(spec, seed):
    if spec[0] == "jet":
        c = fixtures.make_case(spec[1], spec[2], 30.0, 15.0, 1.2, 2000.0, sc=True, dt_mode=1)
    else:
        wall = NSCBC_NOSLIP_WALL if spec[4] % 2 else SAT_NOSLIP_WALL
        c = fixtures.nozzle_case(Nz=spec[1], Nr=spec[2], iw=spec[3], jb=spec[4], jt=spec[5], wall=wall, sc=True, Mj=1.2,
                                 Re=2000.0, dt_mode=1)
    rng = np.random.default_rng(seed)
    for e in (0, 1, 3, 4):
        c["pv"][e] += 0.01 * rng.standard_normal(c["pv"][e].shape)
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("spec", CASES, ids=lambda s: "-".join(map(str, s)))
def test_rhs_against_oracle(oracle_mod, spec):
    c = _case(spec, 11)
    p = axj.patches_from_records(c["records"], c["Nz"], c["Nr"])
    dev = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
    ora = oracle_mod.Oracle(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
    dev.set_state(c["pv"], c["target"])
    ora.set_state(c["pv"], c["target"])
    a, b = dev.compute_rhs(c["pv"]), ora.compute_rhs(c["pv"])
    v = max(np.abs(b[k]).max() for k in (1, 2, 3))
    for k in range(5):
        scale = v if k in (1, 2, 3) else np.abs(b[k]).max()
        assert np.abs(a[k] - b[k]).max() <= REL * scale, k
    dev.close()
