"""Inputs outside the range in which the FP32 estimate of the screened time-step scan bounds a
point's rate: the scan has to evaluate such points in FP64, on grids large enough to be screened
as on small ones. Oracle: the formula of ModInputOutput.f90:395-416 over every point in NumPy (64
bits). Tolerance: as for the scan itself, 1e-14 (a rate is a sum of three terms of at most eight
roundings each, plus a power within 2 ulp; the difference lambda = 0.6 mu - 2/3 mu loses one
digit of its part)."""
import ctypes as C

import numpy as np
import pytest

import axisymmetricjet_b200 as axj

pytestmark = pytest.mark.gpu
TOL = 1e-14
SIZES = [(257, 13), (450, 311)]  # below and above 98,304 points


def _call(pv, dxidz, detadr, params, stale=1.0):
    import torch
    fn = axj.load_library().axj_compute_dt_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p,
                   C.POINTER(axj.AxjParams), C.c_double, C.c_void_p, C.c_void_p]
    _, Nr, Nz = pv.shape
    d, x, y = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pv, dxidz, detadr))
    dt = torch.zeros(1, dtype=torch.float64, device="cuda")
    rc = fn(d.data_ptr(), Nz, Nz, Nr, x.data_ptr(), y.data_ptr(), None, C.byref(params), stale, dt.data_ptr(),
            torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return float(dt.item())


def _dts(pv, dxidz, detadr, p, stale=None):
    x, y = dxidz[None, :], detadr[:, None]
    T = pv[4]
    mu = T ** 0.666
    lam = 0.6 * mu - 2.0 / 3.0 * mu
    inv = np.abs(pv[3] * x + pv[1] * y) + np.sqrt(T if stale is None else stale) * np.sqrt(x * x + y * y)
    m = np.maximum(np.maximum(mu / p.Re, lam / p.Re), mu / (p.Re * p.Pr))
    return p.CFL / (inv + 2.0 * m * (np.abs(x) + np.abs(y)) ** 2)


def _flow(Nz, Nr, seed=3):
    rng = np.random.default_rng(seed)
    pv = np.ones((5, Nr, Nz))
    pv[1], pv[3] = rng.standard_normal((2, Nr, Nz))
    pv[4] = rng.uniform(0.3, 3.0, (Nr, Nz))
    return pv, rng.uniform(1.0, 80.0, Nz), rng.uniform(1.0, 200.0, Nr)


@pytest.mark.parametrize("Nz,Nr", SIZES)
@pytest.mark.parametrize("Re,Pr", [(-50.0, 0.72), (50.0, -0.72), (-50.0, -0.72), (-50.0, 100.0)])
def test_negative_reynolds_or_prandtl_number(Nz, Nr, Re, Pr):
    """The viscous part's maximum is then another of its terms than the estimate's."""
    pv, dxidz, detadr = _flow(Nz, Nr)
    p = axj.default_params(dt_mode=1, Re=Re, Pr=Pr)
    want = _dts(pv, dxidz, detadr, p).min()
    assert abs(_call(pv, dxidz, detadr, p) - want) <= TOL * abs(want)


@pytest.mark.parametrize("Nz,Nr", [(48, 40), (450, 311)])
@pytest.mark.parametrize("CFL", [-0.5, 0.0])
def test_handle_without_a_positive_cfl(oracle_mod, Nz, Nr, CFL):
    """dt = CFL / x is then not smallest where x is largest; the two entry points agree."""
    from axisymmetricjet_b200 import fixtures
    c = fixtures.make_case(Nz, Nr, 30.0, 15.0, 0.9, 1000.0, dt_mode=1, CFL=CFL)
    c["pv"][1] += 0.1 * np.random.default_rng(3).standard_normal((Nr, Nz))
    p = axj.patches_from_records(c["records"], Nz, Nr)
    with axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"], p) as s:
        ora = oracle_mod.Oracle(c["params"], c["zvec"], c["rvec"], c["ibval"], p)
        s.set_state(c["pv"], c["target"])
        ora.set_state(c["pv"], c["target"])
        want = ora.compute_time_step()
        assert abs(s.compute_time_step() - want) <= TOL * abs(want)
        mz, mr = ora.metrics()[:2]
        got = _call(c["pv"], np.ascontiguousarray(mz[0]), np.ascontiguousarray(mr[:, 0]), c["params"])
        assert abs(got - want) <= TOL * abs(want)


@pytest.mark.parametrize("Nz,Nr", SIZES)
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("T", [-1e-40, -1e-300])
def test_small_negative_temperature(Nz, Nr, mode, T):
    """T**0.666 of a negative T is not a number, however small it is."""
    pv, dxidz, detadr = _flow(Nz, Nr)
    p = axj.default_params(dt_mode=mode)
    assert _call(pv, dxidz, detadr, p) > 0.0
    pv[4, Nr // 2, Nz // 3] = T
    assert np.isnan(_call(pv, dxidz, detadr, p))


@pytest.mark.parametrize("Nz,Nr", SIZES)
@pytest.mark.parametrize("kind", ["metrics", "temperature", "viscosity", "velocity", "no sound"])
def test_below_single_precision(Nz, Nr, kind):
    """Rates whose parts are below FP32's normal range."""
    pv, dxidz, detadr = _flow(Nz, Nr)
    p, stale = axj.default_params(dt_mode=1), None
    if kind == "metrics":  # lengths of 1e19 units
        dxidz, detadr = np.full(Nz, 5e-20), np.zeros(Nr)
        pv[3] = 0.5
        pv[4] = 1.0
        pv[3, Nr // 2, Nz // 3], pv[4, Nr // 2, Nz // 3] = 0.4, 9.0
    elif kind == "temperature":
        pv[1] = pv[3] = 0.0
        pv[4] *= 1e-40
    elif kind == "viscosity":
        pv[1] = pv[3] = 0.0
        p, stale = axj.default_params(dt_mode=0, Re=1e44), 0.0
    elif kind == "no sound":  # the stale T before the first step
        pv[1] = pv[3] = 0.0
        p, stale = axj.default_params(dt_mode=0), 0.0
    else:  # an advection rate of order one from a velocity below and a metric far above
        pv[1] = 0.0
        pv[3] *= 1e-45
        p, stale = axj.default_params(dt_mode=0, Re=1e300), 0.0
        dxidz, detadr = dxidz * 1e36, detadr * 1e-3
    want = _dts(pv, dxidz, detadr, p, stale).min()
    got = _call(pv, dxidz, detadr, p, 1.0 if stale is None else stale)
    assert abs(got - want) <= TOL * want


@pytest.mark.parametrize("Nz,Nr", [(1, 98305), (4, 100000), (10, 60000), (11, 196608), (11, 196609), (12, 49152),
                                   (12, 49153), (16, 12289), (31, 3300), (33, 4500), (33, 7000), (65, 1513)])
def test_narrow_grids(Nz, Nr):
    """Grids either side of the rule that screens rows of few columns only above more points."""
    pv, dxidz, detadr = _flow(Nz, Nr, Nz + Nr)
    p = axj.default_params(dt_mode=1)
    want = _dts(pv, dxidz, detadr, p).min()
    assert abs(_call(pv, dxidz, detadr, p) - want) <= TOL * want
