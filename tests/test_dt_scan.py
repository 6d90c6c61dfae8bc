"""The screened point scan of ComputeTimeStep: FP32 estimates choose the points whose rate is
evaluated in FP64. The result must be the full scan's minimum wherever the largest rate sits
and however near the other points come to it. Oracle: the formula of ModInputOutput.f90:395-416
over every point in NumPy (64 bits).

Tolerance: a rate is a sum of three positive terms of at most eight roundings each (the
advection term's inputs are random or make it exact) plus a power within 2 ulp on either side:
below 24 * 1.1e-16 < 1e-14. The near ties differ by
1e-6 to 1e-3, so a wrongly screened point shows."""
import ctypes as C

import numpy as np
import pytest

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures

pytestmark = pytest.mark.gpu
TOL = 1e-14


def _rates(pv, dxidz, detadr, p, stale=None):
    x, y = dxidz[None, :], detadr[:, None]
    T = pv[4]
    mu = T ** 0.666
    inv = np.abs(pv[3] * x + pv[1] * y) + np.sqrt(T if stale is None else stale) * np.sqrt(x * x + y * y)
    return inv + 2.0 * np.maximum(mu / p.Re, mu / (p.Re * p.Pr)) * (np.abs(x) + np.abs(y)) ** 2


def _fields(Nz, Nr, kind, seed):
    rng = np.random.default_rng(seed)
    pv = np.zeros((5, Nr, Nz))
    pv[0] = 1.0
    pv[4] = 1.0
    if kind == "random":
        pv[1], pv[3] = rng.standard_normal((2, Nr, Nz))
        pv[4] = rng.uniform(0.3, 3.0, (Nr, Nz))
    elif kind == "ties":  # every point within 1e-6 of the largest
        pv[3] = 0.5 * (1.0 + 1e-6 * rng.random((Nr, Nz)))
    else:
        # cancelling advection terms (the estimate's error is relative to its parts): multiples
        # of 2**-20 below 2**14, so that their products with a metric of 16 and their sum are
        # exact in 64 bits, whatever the order or contraction
        pv[3] = np.round(1e4 * (1.0 + 1e-3 * rng.random((Nr, Nz))) * 2.0 ** 20) / 2.0 ** 20
        pv[1] = -np.round(pv[3] * (1.0 + 1e-5 * rng.random((Nr, Nz))) * 2.0 ** 20) / 2.0 ** 20
    return pv


def _noalloc(pv, dxidz, detadr, params, ib=None, stale=1.0, pad=5):
    import torch
    lib = axj.load_library()
    fn = lib.axj_compute_dt_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_int64, C.c_int64, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p,
                   C.POINTER(axj.AxjParams), C.c_double, C.c_void_p, C.c_void_p]
    _, Nr, Nz = pv.shape
    buf = np.full((5, Nr, Nz + pad), np.nan)
    buf[..., :Nz] = pv
    d = torch.from_numpy(buf).cuda()
    b = None
    if ib is not None:
        bb = np.zeros((Nr, Nz + pad))
        bb[:, :Nz] = ib
        b = torch.from_numpy(bb).cuda()
    x, y = torch.from_numpy(dxidz).cuda(), torch.from_numpy(detadr).cuda()
    dt = torch.zeros(1, dtype=torch.float64, device="cuda")
    rc = fn(d.data_ptr(), Nz + pad, Nz, Nr, x.data_ptr(), y.data_ptr(), b.data_ptr() if b is not None else None,
            C.byref(params), stale, dt.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return float(dt.item())


# below, at and above the size from which the scan is screened (98,304 points), rows shorter
# and longer than a block, ragged last chunks
SIZES = [(1, 1), (12, 13), (255, 9), (4400, 7), (1536, 64), (1537, 64), (4737, 64), (13, 23317), (257, 1283), (4400, 160),
         (1, 2097153), (33, 270000)]  # the last two: more strips than the scratch has places


@pytest.mark.parametrize("Nz,Nr", SIZES)
@pytest.mark.parametrize("kind", ["random", "ties", "cancel"])
@pytest.mark.parametrize("mode", [0, 1])
def test_scan_equals_full_scan(Nz, Nr, kind, mode):
    rng = np.random.default_rng(Nz + 7 * Nr)
    one = kind != "random"
    dxidz = np.full(Nz, 16.0) if one else rng.uniform(1.0, 80.0, Nz)
    detadr = np.full(Nr, 16.0) if one else rng.uniform(1.0, 200.0, Nr)
    p = axj.default_params(dt_mode=mode, Re=1000.0)
    for seed in range(3):
        pv = _fields(Nz, Nr, kind, seed)
        want = p.CFL / _rates(pv, dxidz, detadr, p, None if mode else 1.0).max()
        got = _noalloc(pv, dxidz, detadr, p)
        assert abs(got - want) <= TOL * want, (seed, got, want)


def test_scan_blanked_negative_cfl_and_non_finite():
    Nz, Nr = 1030, 307
    rng = np.random.default_rng(5)
    dxidz, detadr = rng.uniform(1.0, 80.0, Nz), rng.uniform(1.0, 200.0, Nr)
    p = axj.default_params(dt_mode=1)
    pv = _fields(Nz, Nr, "random", 1)
    x = _rates(pv, dxidz, detadr, p)
    ib = np.ones((Nr, Nz))
    ib[x > np.quantile(x, 0.9)] = 0.0  # the largest rates are blanked
    want = p.CFL / x[ib == 1.0].max()
    assert abs(_noalloc(pv, dxidz, detadr, p, ib) - want) <= TOL * want
    assert _noalloc(pv, dxidz, detadr, p, 0.0 * ib) == 100.0
    q = axj.default_params(dt_mode=1, CFL=-0.5)  # the smallest dt is then the smallest rate's
    want = -0.5 / x.min()
    assert abs(_noalloc(pv, dxidz, detadr, q) - want) <= TOL * abs(want)
    for e in (1, 3, 4):
        for bad in (np.nan, np.inf, -np.inf):
            v = pv.copy()
            v[e, 20, 77] = bad
            assert np.isnan(_noalloc(v, dxidz, detadr, p)), (e, bad)
            assert np.isnan(_noalloc(v, dxidz, detadr, axj.default_params(dt_mode=0))), (e, bad)


@pytest.mark.parametrize("Nz,Nr", [(48, 40), (1300, 245)])
def test_handle_scan_forgets_the_previous_state(Nz, Nr):
    """The bound of one state must not screen the next: a fast state, then a slow one."""
    c = fixtures.make_case(Nz, Nr, 30.0, 15.0, 0.9, 1000.0, dt_mode=1)
    s = axj.AxiJetSolver(c["params"], c["zvec"], c["rvec"], c["ibval"],
                         axj.patches_from_records(c["records"], Nz, Nr))
    tables = axj.operator_tables()
    import restatement
    mz, mr, _, _ = restatement.metrics(tables[0], c["z"], c["r"])
    dts = []
    for scale in (50.0, 1.0, 0.02):
        pv = c["pv"].copy()
        pv[1] += 0.01 * np.random.default_rng(3).standard_normal((Nr, Nz))
        pv[1] *= scale
        pv[3] *= scale
        pv[4] *= scale
        s.set_state(pv, c["target"])
        want = c["params"].CFL / _rates(pv, mz[0], mr[:, 0], c["params"]).max()
        got = s.compute_time_step()
        assert abs(got - want) <= TOL * want, (scale, got, want)
        dts.append(got)
    assert dts[0] < dts[1] < dts[2]
    s.close()
