"""RK4's last sum from the three stage states (the FP64 path's: differences to pv_old) against
the running sum it stands for, each against extended precision: the rounding error of a step is
no larger. The sums are restated here as the stage kernel forms them (round to nearest, no FMA)."""
import numpy as np
import pytest


def running_sum(u, k):
    a = u + (1.0 / 6.0) * k[0]
    a = a + (1.0 / 3.0) * (k[1] + k[2])
    return a + (1.0 / 6.0) * k[3]


def stage_states(u, k):
    u1, u2, u3 = u + 0.5 * k[0], u + 0.5 * k[1], u + k[2]
    q = ((u1 - u) + (u3 - u)) + 2.0 * (u2 - u)
    return u + ((1.0 / 3.0) * q + (1.0 / 6.0) * k[3])


@pytest.mark.parametrize("scale", [1e-1, 1e-3, 1e-6, 1e-12])
def test_rounding_error_of_a_step_is_no_larger(scale):
    L = np.longdouble
    assert np.finfo(L).nmant > 60
    rng = np.random.default_rng(3)
    u = rng.uniform(0.5, 2.0, 200000)
    k = [scale * rng.standard_normal(u.size) for _ in range(4)]
    exact = L(u) + L(k[0]) / 6 + (L(k[1]) + L(k[2])) / 3 + L(k[3]) / 6
    err = [float(np.sqrt(np.mean(((L(f(u, k)) - exact) / np.spacing(u)) ** 2))) for f in (running_sum, stage_states)]
    assert err[1] <= err[0], err
    assert err[1] < 0.45, err  # 0.50 and 0.37 units in the last place
