"""The page-locked places of the handles' step scalars: more handles than one page holds, made,
stepped by the host and closed by several threads in different orders, give what a handle of its
own gives, bit for bit."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures


def _solver(c):
    s = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"],
                         axj.patches_from_records(c["records"], c["Nz"], c["Nr"]))
    s.set_state(c["pv"], c["target"])
    return s


def _steps(s, scale):
    dts = []
    for _ in range(3):
        dts.append(s.compute_time_step())
        s.rk4(scale * dts[-1])
    return dts, s.get_time(), s.get_state()


@pytest.mark.gpu
def test_many_handles_and_threads():
    c = fixtures.make_case(48, 40, 30.0, 15.0, 0.9, 1000.0, dt_mode=1)
    scales = [1.0 - 0.01 * k for k in range(20)]
    with _solver(c) as s:
        alone = []
        for f in scales:
            s.set_state(c["pv"], c["target"])
            alone.append(_steps(s, f))

    def work(t):
        solvers = [_solver(c) for _ in range(20)]
        out = [_steps(s, f) for s, f in zip(solvers, scales)]
        for k in np.random.default_rng(t).permutation(20):
            solvers[k].close()
        return out

    with ThreadPoolExecutor(4) as ex:
        for out in ex.map(work, range(4)):
            for a, b in zip(out, alone):
                assert a[0] == b[0] and a[1] == b[1] and np.array_equal(a[2], b[2])
