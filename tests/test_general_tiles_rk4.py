"""RK4 steps over general stage tiles, unconditionally: the 512-thread form (up to 148 tiles) and the
256-thread form, closure, centred and blanked rows in one warp, wall and forcing terms, with and without shock
capturing. Against the CPU oracle, whose own state is asserted finite and bounded first.

Tolerance: the FP64 bars, 1e-12 of each field's largest value (velocities share one scale)."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures
from axisymmetricjet_b200._ffi import NSCBC_NOSLIP_WALL, SAT_NOSLIP_WALL

REL = 1e-12
# 33 columns over 1200 rows: the shock-capturing step of that grid is stable at a far smaller dt only
CASES = [("jet", 70, 30, 0.2), ("jet", 2300, 16, 0.2), ("jet", 2368, 17, 0.2), ("jet", 2401, 16, 0.2),
         ("jet", 33, 1200, 1e-3), ("nozzle", 61, 70, 9, 20, 26, 0.2), ("nozzle", 2300, 40, 700, 12, 17, 0.2)]


def case(spec, sc):
    kw = dict(sc=sc, dt_mode=1, control_forcing=1, forcing_z0=3.0, forcing_r0=0.5, forcing_lz=1.0, forcing_lr=0.3,
              forcing_mat=np.arange(25.0).reshape(5, 5) * 1e-3)
    if spec[0] == "jet":
        return fixtures.make_case(spec[1], spec[2], 30.0, 15.0, 0.9, 1000.0, **kw)
    return fixtures.nozzle_case(Nz=spec[1], Nr=spec[2], iw=spec[3], jb=spec[4], jt=spec[5],
                                wall=SAT_NOSLIP_WALL if sc else NSCBC_NOSLIP_WALL, **kw)


def oracle_steps(ora, factor):
    """Two steps; their dts and the state."""
    dts = []
    for _ in range(2):
        dts.append(factor * ora.compute_time_step())
        ora.rk4(dts[-1])
    out = ora.get_state()
    assert np.isfinite(out).all() and np.abs(out).max() < 10.0
    return dts, out


@pytest.mark.gpu
@pytest.mark.parametrize("sc", [False, True])
@pytest.mark.parametrize("spec", CASES, ids=lambda s: "-".join(map(str, s)))
def test_two_steps_against_oracle(oracle_mod, spec, sc):
    c = case(spec, sc)
    p = axj.patches_from_records(c["records"], c["Nz"], c["Nr"])
    ora = oracle_mod.Oracle(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
    ora.set_state(c["pv"], c["target"])
    dts, b = oracle_steps(ora, spec[-1])
    with axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"], p) as dev:
        dev.set_state(c["pv"], c["target"])
        for dt in dts:
            dev.rk4(dt)
        a = dev.get_state()
    v = max(np.abs(b[k]).max() for k in (1, 2, 3))
    for k in range(5):
        scale = v if k in (1, 2, 3) else np.abs(b[k]).max()
        assert np.abs(a[k] - b[k]).max() <= REL * scale, k
