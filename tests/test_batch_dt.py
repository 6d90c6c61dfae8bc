"""The batched time step over grids of both kinds of scan in one FP64 batch: instances below the
size that is screened, at it (98,304 points) and above, and a narrow one, against individual runs.

Tolerance: 1e-12 of each field's largest value and of the time, the FP64 bar of a batch against its
handles."""
import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures

REL = 1e-12
GRIDS = [(48, 40), (256, 384), (1300, 245), (13, 3000), (450, 311)]


def _solvers():
    out = []
    for k, (Nz, Nr) in enumerate(GRIDS):
        c = fixtures.make_case(Nz, Nr, 30.0, 15.0, 0.9, 1000.0, dt_mode=1, seed=k, CFL=1e-3 if Nz == 13 else 0.4)
        s = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"], axj.patches_from_records(c["records"], Nz, Nr))
        s.set_state(c["pv"], c["target"])
        out.append(s)
    return out


@pytest.mark.gpu
def test_batch_of_both_scans_equals_individual_runs():
    alone, together = _solvers(), _solvers()
    for s in alone:
        s.run(4)
    batch = axj.AxjBatch(together)
    batch.run(4)
    for s, t in zip(alone, together):
        (ia, ta), (ib, tb) = s.get_time(), t.get_time()
        assert ia == ib and abs(ta - tb) <= REL * ta
        a, b = s.get_state(), t.get_state()
        assert np.isfinite(a).all()
        for e in range(5):
            assert np.abs(a[e] - b[e]).max() <= REL * max(np.abs(a[e]).max(), np.abs(a[3]).max())
    batch.close()
    for s in alone + together:
        s.close()
