"""General stage tiles either side of the size from which two of their CTAs share an SM (148
tiles), and warps whose points mix centred, closure and blanked rows in both directions, with and
without shock capturing: ComputeRHS and one RK4 step against the CPU oracle.

Tolerance: the FP64 bars, 1e-12 of each field's largest value (velocities share one scale)."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures
from axisymmetricjet_b200._ffi import NSCBC_NOSLIP_WALL, SAT_NOSLIP_WALL

REL = 1e-12
# tiles: 2 bands x Nz / 32 (thin rows) or the z faces, bands and walls of a nozzle
CASES = [("jet", 70, 30), ("jet", 2300, 16), ("jet", 2368, 17), ("jet", 2401, 16), ("jet", 33, 1200),
         ("nozzle", 61, 70, 9, 20, 26), ("nozzle", 2300, 40, 700, 12, 17)]


@pytest.mark.gpu
@pytest.mark.parametrize("sc", [False, True])
@pytest.mark.parametrize("spec", CASES, ids=lambda s: "-".join(map(str, s)))
def test_against_oracle(oracle_mod, spec, sc):
    kw = dict(sc=sc, dt_mode=1, control_forcing=1, forcing_z0=3.0, forcing_r0=0.5, forcing_lz=1.0, forcing_lr=0.3,
              forcing_mat=np.arange(25.0).reshape(5, 5) * 1e-3)
    if spec[0] == "jet":
        c = fixtures.make_case(spec[1], spec[2], 30.0, 15.0, 0.9, 1000.0, **kw)
    else:
        c = fixtures.nozzle_case(Nz=spec[1], Nr=spec[2], iw=spec[3], jb=spec[4], jt=spec[5],
                                 wall=SAT_NOSLIP_WALL if sc else NSCBC_NOSLIP_WALL, **kw)
    p = axj.patches_from_records(c["records"], c["Nz"], c["Nr"])
    dev = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
    ora = oracle_mod.Oracle(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
    dev.set_state(c["pv"], c["target"])
    ora.set_state(c["pv"], c["target"])

    def close(a, b):
        v = max(np.abs(b[k]).max() for k in (1, 2, 3))
        for k in range(5):
            scale = v if k in (1, 2, 3) else np.abs(b[k]).max()
            assert np.abs(a[k] - b[k]).max() <= REL * max(scale, 1e-300), k

    close(dev.compute_rhs(c["pv"]), ora.compute_rhs(c["pv"]))
    dt = 0.2 * dev.compute_time_step()
    ora.rk4(dt)
    if np.abs(ora.get_state()).max() < 10.0:  # not where the oracle's own step is unstable (33 x 1200 with sc)
        dev.rk4(dt)
        close(dev.get_state(), ora.get_state())
    dev.close()
