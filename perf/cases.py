"""Performance cases of the framework: what a program that drives it spends its time on.

A case is a dict of plain values. `listed()` names the standing ones, `draw(rng)` gives
another of the same ranges, `prepare(case, seed)` makes what a program has in hand before
the call, `run(state)` is one pass through the public entry points with its outputs,
`work(case)` the bytes and operations the path cannot do without, and `exact(case, seed)`
the same outputs in 64-bit PyTorch from the published formulas, without the framework.

Kinds of passes
  advance   hand the solver a solution and its target in pinned host memory, advance it
            `steps` steps on the device (dt kept there), read the solution back: the
            segment between two outputs or restarts of a run
  driver    the same with the host's own step loop: ComputeTimeStep, dt read back, RK4
  batch     the same for many uneven jets advanced together by one batch
  dt        ComputeTimeStep on device arrays that the caller owns
  train     one training run of the learned sensor's network on a device data set

Runs in mixed precision (FP32 stage states and stencils) write their solution in single
precision, the precision their stage arithmetic has; plain runs write 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

import axisymmetricjet_b200 as axj
from axisymmetricjet_b200 import fixtures
from axisymmetricjet_b200.train_sensor import load_model

DEFAULTS = dict(zmax=30.0, rmax=15.0, mach=1.5, re=5000.0, sc=True, precision=0, sensor=0, judge_every=50,
                judge_stages=0, dt_mode=1, forcing=0, nozzle=0)


def listed():
    return [
        # latency: a small shock-capturing jet driven step by step by the host program,
        # as the Fortran driver's loop does (dt to the host every step)
        dict(name="driver_96x64", kind="driver", Nz=96, Nr=64, steps=20, dt_mode=0),
        # the small plain jet (no shock capturing), the configured 100 steps
        dict(name="plain_512x128", kind="advance", Nz=512, Nr=128, steps=100, rmax=10.0, mach=0.9, re=1000.0,
             sc=False, dt_mode=0),
        # a nozzle with its lip blanked, wall patches and feedback forcing on a ragged grid
        dict(name="nozzle_787x203", kind="advance", Nz=787, Nr=203, steps=60, mach=0.9, re=1000.0, nozzle=94,
             forcing=1),
        # a mid-sized jet of odd extents, plain FP64 with shock capturing
        dict(name="jet_1801x333", kind="advance", Nz=1801, Nr=333, steps=60),
        # the production jet: plain FP64 ...
        dict(name="jet_4400x640", kind="advance", Nz=4400, Nr=640, steps=50, zmax=60.0, dt_mode=0),
        # ... in mixed precision ...
        dict(name="mixed_4400x640", kind="advance", Nz=4400, Nr=640, steps=100, zmax=60.0, precision=1),
        # ... and with the learned sensor between its judge steps
        dict(name="learned_4400x640", kind="advance", Nz=4400, Nr=640, steps=100, zmax=60.0, precision=1, sensor=1),
        # uneven jets with harmonic inflow forcing advanced together, mixed precision
        dict(name="batch_12", kind="batch", instances=12, sizes=2024, steps=40, precision=1, rmax=10.0),
        # a batch of a few small jets in plain FP64
        dict(name="batch_4_fp64", kind="batch", instances=4, sizes=7, steps=20, precision=0, rmax=10.0),
        # ComputeTimeStep alone on a caller's device arrays
        dict(name="dt_4400x640", kind="dt", Nz=4400, Nr=640, zmax=60.0),
        # training of the learned sensor's network
        dict(name="train_65536", kind="train", Nz=1024, Nr=256, snapshots=4, steps=20, batch=65536),
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advance"] * 6 + ["driver", "batch", "batch", "dt", "train"])
    if kind == "driver":
        return dict(kind=kind, Nz=_spread(rng, 64, 512), Nr=_spread(rng, 48, 160), steps=rng.randint(5, 20),
                    precision=rng.randint(0, 1), dt_mode=rng.randint(0, 1), mach=round(rng.uniform(0.9, 1.5), 3))
    if kind == "batch":
        return dict(kind=kind, instances=rng.randint(3, 12), sizes=rng.randint(1, 9999), steps=rng.randint(8, 20),
                    precision=rng.randint(0, 1), sensor=rng.choice([0, 0, 2]), judge_every=rng.choice([5, 50]),
                    rmax=10.0)
    if kind == "dt":
        return dict(kind=kind, Nz=_spread(rng, 256, 4400), Nr=_spread(rng, 128, 640), zmax=60.0,
                    dt_mode=rng.randint(0, 1))
    if kind == "train":
        return dict(kind=kind, Nz=_spread(rng, 256, 1024), Nr=_spread(rng, 64, 256), snapshots=rng.randint(2, 4),
                    steps=rng.randint(10, 20), batch=_spread(rng, 2048, 65536))
    case = dict(kind=kind, Nz=_spread(rng, 128, 4400), Nr=_spread(rng, 64, 640), steps=rng.randint(15, 40),
                mach=round(rng.uniform(0.9, 1.5), 3), re=round(rng.uniform(1000.0, 5000.0), 1),
                precision=rng.randint(0, 1), dt_mode=rng.randint(0, 1))
    case["zmax"] = 60.0 if case["Nz"] > 2048 else 30.0
    form = rng.choice(["plain", "sc", "sc", "sc", "learned", "held", "nozzle"])
    if form == "plain":
        case.update(sc=False, forcing=rng.randint(0, 1))
    elif form in ("learned", "held"):
        case.update(sensor=1 if form == "learned" else 2, judge_every=rng.choice([10, 50]),
                    judge_stages=rng.choice([0, 1]))
        if form == "learned":
            case["precision"] = 1  # the network's BF16 goes with the mixed form
    elif form == "nozzle":
        case.update(nozzle=rng.choice([93, 94]), mach=0.9, re=1000.0, sc=rng.random() < 0.5, dt_mode=1)
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _full(case):
    return {**DEFAULTS, **case}


def _fixture(case, seed, **over):
    """The fixture dict of a flow case: grid, iblank, bc records, parameters, solution
    and target."""
    c = {**_full(case), **over}
    pkw = dict(precision=c["precision"], sensor=c["sensor"], judge_every=c["judge_every"],
               judge_stages=c["judge_stages"], dt_mode=c["dt_mode"])
    if c["forcing"] == 1:
        # feedback of V_r on V_z in a Gaussian window inside the shear layer
        pkw.update(control_forcing=1, forcing_alpha=0.5, forcing_z0=8.0, forcing_r0=0.5, forcing_lz=1.0,
                   forcing_lr=0.3)
    elif c["forcing"] == 2:
        # harmonic inflow forcing in the shear layer near the inflow
        pkw.update(control_forcing=2, forcing_z0=1.0, forcing_r0=0.5, forcing_lz=0.5, forcing_lr=0.2,
                   harmonic_amp=c["amp"] * c["mach"], harmonic_st=c["st"], harmonic_uj=c["mach"])
    if c["nozzle"]:
        r = c["rmax"] * np.sinh(3.0 * np.arange(c["Nr"]) / (c["Nr"] - 1)) / np.sinh(3.0)
        jb = int(np.searchsorted(r, 1.0)) + 1
        out = fixtures.nozzle_case(Nz=c["Nz"], Nr=c["Nr"], zmax=c["zmax"], rmax=c["rmax"], Mj=c["mach"], Re=c["re"],
                                   iw=c["Nz"] // 7, jb=jb, jt=jb + max(5, c["Nr"] // 38), wall=c["nozzle"],
                                   sc=c["sc"], seed=seed, **pkw)
    else:
        out = fixtures.make_case(c["Nz"], c["Nr"], c["zmax"], c["rmax"], c["mach"], c["re"], sc=c["sc"], seed=seed,
                                 **pkw)
    if c["forcing"] == 1:
        out["params"].forcing_mat[3 * 5 + 1] = 1.0
    return out


def _batch_fixtures(case, seed):
    """The uneven jets of a batch: extents, Mach, Reynolds and forcing by the case, the
    perturbations of their solutions by the seed."""
    c = _full(case)
    rng = np.random.default_rng(c["sizes"])
    out = []
    for k in range(c["instances"]):
        over = dict(Nz=int(32 * np.round(rng.uniform(256, 2048) / 32)), Nr=int(32 * np.round(rng.uniform(96, 384) / 32)),
                    mach=float(rng.uniform(0.9, 1.5)), re=float(rng.uniform(1000.0, 5000.0)), forcing=2,
                    amp=float(rng.uniform(0.0, 0.02)), st=float(rng.uniform(0.2, 0.6)))
        out.append(_fixture(case, seed + k, **over))
    return out


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _solver(f, sensor=0):
    s = axj.AxiJetSolver(f["params"], f["zvec"], f["rvec"], f["ibval"],
                         axj.patches_from_records(f["records"], f["Nz"], f["Nr"]))
    if sensor == 1:
        s.mlp_set(load_model())
    return s


def _flow_state(f, sensor):
    s = dict(solver=_solver(f, sensor), pv=_pinned(f["pv"]), target=_pinned(f["target"]),
             out=_pinned(np.empty_like(f["pv"])))
    if f["params"].precision:
        s["out32"] = np.empty(f["pv"].shape, dtype=np.float32)
    return s


def prepare(case, seed):
    c = _full(case)
    if c["kind"] in ("advance", "driver"):
        return dict(_flow_state(_fixture(case, seed), c["sensor"]), case=c)
    if c["kind"] == "batch":
        parts = [_flow_state(f, c["sensor"]) for f in _batch_fixtures(case, seed)]
        for p in parts:
            p["solver"].set_state(p["pv"], p["target"])
        batch = axj.AxjBatch([p["solver"] for p in parts])
        batch.autotune(3)  # as a batch's owner does once before its run
        return dict(batch=batch, parts=parts, case=c)
    if c["kind"] == "dt":
        return _dt_state(c, seed)
    return _train_state(c, seed)


def _dt_fixture(c, seed):
    """A jet whose flow is perturbed everywhere, as some way into a run."""
    f = _fixture(c, seed)
    noise = np.random.default_rng(seed).standard_normal((c["Nr"], c["Nz"]))
    for e in (1, 3, 4):
        f["pv"][e] += 1e-3 * noise
    return f


def _dt_state(c, seed):
    """A caller's device arrays: the solution in rows of a pitch of its own, the 1-D
    metrics, and the result's place."""
    f = _dt_fixture(c, seed)
    pitch = c["Nz"] + 24
    pv = torch.zeros((5, c["Nr"], pitch), dtype=torch.float64, device="cuda")
    pv[:, :, :c["Nz"]] = torch.from_numpy(f["pv"]).cuda()
    lib = axj.load_library()
    fn = lib.axj_compute_dt_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p,
                   ctypes.c_void_p, ctypes.POINTER(axj.AxjParams), ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p]
    return dict(case=c, fn=fn, params=f["params"], pv=pv, pitch=pitch, dt=torch.zeros(1, dtype=torch.float64, device="cuda"),
                dxidz=torch.from_numpy(1.0 / _metric(f["z"])).cuda(), detadr=torch.from_numpy(1.0 / _metric(f["r"])).cuda())


def _train_state(c, seed):
    """A handle whose data set holds snapshots of a jet some steps apart, and the seeded
    initial model."""
    f = _fixture(c, seed)
    s = _solver(f)
    s.set_state(f["pv"], f["target"])
    s.dataset_reserve(c["snapshots"])
    for _ in range(c["snapshots"]):
        s.run(10)
        s.dataset_add()
    return dict(case=c, solver=s, model=axj.mlp_init(seed), seed=seed)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _solution(s):
    pv = s["solver"].get_state(s["out"])
    if "out32" in s:
        np.copyto(s["out32"], pv, casting="same_kind")
        return s["out32"]
    return pv


def run(state):
    c = state["case"]
    if c["kind"] == "advance":
        s = state["solver"]
        s.set_state(state["pv"], state["target"])
        dt = s.run(c["steps"])
        return {"pv": _solution(state), "dt": dt}
    if c["kind"] == "driver":
        s = state["solver"]
        s.set_state(state["pv"], state["target"])
        for _ in range(c["steps"]):
            dt = s.compute_time_step()
            s.rk4(dt)
        return {"pv": _solution(state), "dt": dt}
    if c["kind"] == "batch":
        for p in state["parts"]:
            p["solver"].set_state(p["pv"], p["target"])
        state["batch"].run(c["steps"])
        return [_solution(p) for p in state["parts"]]
    if c["kind"] == "dt":
        rc = state["fn"](state["pv"].data_ptr(), state["pitch"], c["Nz"], c["Nr"], state["dxidz"].data_ptr(),
                         state["detadr"].data_ptr(), None, ctypes.byref(state["params"]), 1.0, state["dt"].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise axj.AxjError(rc, "axj_compute_dt_noalloc")
        return state["dt"]
    s = state["solver"]
    s.mlp_set(state["model"])
    loss = s.mlp_train(steps=c["steps"], batch=c["batch"], seed=state["seed"], fit_normalization=1)
    return {"loss": loss, "model": s.mlp_get()}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c = _full(case)
    if c["kind"] == "train":
        # forward, input and weight gradients of 100 -> 64 -> 64 -> 2; the gathered windows
        mac = 2 * (100 * 64) + 3 * (64 * 64 + 64 * 2)
        return {"bytes": c["steps"] * c["batch"] * (100 + 2) * 4, "flops": 2 * mac * c["steps"] * c["batch"]}
    if c["kind"] == "dt":
        return {"bytes": 24 * c["Nz"] * c["Nr"], "flops": 60 * c["Nz"] * c["Nr"]}
    if c["kind"] == "batch":
        rng = np.random.default_rng(c["sizes"])
        pts = 0
        for _ in range(c["instances"]):
            pts += int(32 * np.round(rng.uniform(256, 2048) / 32)) * int(32 * np.round(rng.uniform(96, 384) / 32))
            rng.uniform(size=4)
    else:
        pts = c["Nz"] * c["Nr"]
    # 17 accesses of the five fields per RK4 step; in mixed precision the three stage
    # states (written and read once each) are 4-byte; plus the solution and target in, the solution out
    per_step = 5 * (11 * 8 + 6 * (4 if c["precision"] else 8))
    ops = 4 * (700 + (300 if c["sc"] else 0))
    return {"bytes": pts * (per_step * c["steps"] + 120), "flops": pts * ops * c["steps"]}


# ---------------------------------------------------------------------------
# the same in 64 bits: dense line operators in PyTorch
# ---------------------------------------------------------------------------
def _mirrored(rows, width, sign):
    t = np.zeros((9, width))
    for k, row in enumerate(rows):
        t[k, :len(row)] = row
        t[8 - k] = sign * t[k, ::-1]
    return t


# first- and second-derivative summation-by-parts rows (0-3 and 5-8 closures, 4 centred)
SBP1 = _mirrored([[-24 / 17, 59 / 34, -4 / 17, -3 / 34], [-1 / 2, 0, 1 / 2], [4 / 43, -59 / 86, 0, 59 / 86, -4 / 43],
                  [3 / 98, 0, -59 / 98, 0, 32 / 49, -4 / 49]], 6, -1.0)
SBP2 = _mirrored([[2, -5, 4, -1], [1, -2, 1], [-4 / 43, 59 / 43, -110 / 43, 59 / 43, -4 / 43],
                  [-1 / 49, 0, 59 / 49, -118 / 49, 64 / 49, -4 / 49]], 6, 1.0)
SBP1[4, :5] = [1 / 12, -2 / 3, 0, 2 / 3, -1 / 12]
SBP2[4, :5] = [-1 / 12, 4 / 3, -5 / 2, 4 / 3, -1 / 12]
# truncated-Gaussian filter; the boundary rows are single-precision literals
_F32 = lambda *v: [float(np.float32(x)) for x in v]  # noqa: E731
TGF = _mirrored([[1.0],
                 _F32(0.085777408970, 0.722371828476, 0.356848072173, -0.223119093072, 0.057347064865, 0.000747264596,
                      0.000027453993),
                 _F32(-0.032649010764, 0.143339502575, 0.726678822020, 0.294622121167, -0.186711738069, 0.062038376258,
                      -0.007318073189),
                 _F32(0.000054596010, -0.042124772446, 0.173103107841, 0.700384128648, 0.276543612935, -0.131223506571,
                      0.023424966418, -0.013937561779, 0.024565095706, -0.013098287852, 0.002308621090)], 11, 1.0)
TGF[4, :9] = [107 / 103680, 149 / 12960, 1997 / 25920, 3091 / 12960, 3565 / 10368, 3091 / 12960, 1997 / 25920,
              149 / 12960, 107 / 103680]


def _metric(x):
    """The first-derivative operator, closed at both ends, on one coordinate line."""
    n = len(x)
    out = np.empty(n)
    for i in range(n):
        k, w0, m = (i, 0, 6) if i < 4 else (8 - (n - 1) + i, n - 6, 6) if i >= n - 4 else (4, i - 2, 5)
        out[i] = SBP1[k, :m] @ x[w0:w0 + m]
    return out


def _patches(records, Nz, Nr):
    """0-based inclusive (i0, i1, j0, j1, bc, dir): each face with its four-wide strip."""
    out = []
    for bc, d, i0, i1, j0, j1 in records:
        i0, i1 = (Nz if v == -1 else v for v in (i0, i1))
        j0, j1 = (Nr if v == -1 else v for v in (j0, j1))
        if d == 1:
            i1 = i0 + 3
        elif d == -1:
            i0 = i1 - 3
        elif d == 2:
            j1 = j0 + 3
        else:
            j0 = j1 - 3
        out.append((i0 - 1, i1 - 1, j0 - 1, j1 - 1, bc, d))
    return out


class _Lines:
    """The operators along one direction as dense matrices, one set per distinct pattern
    of stencil rows and blanked points; fields are (..., Nr, Nz)."""

    def __init__(self, codes, blank, along_z):
        self.along_z = along_z
        key = np.where(blank, 9, codes)
        key = key if along_z else key.T
        kinds, self.which = np.unique(key, axis=0, return_inverse=True)
        self.which = self.which.reshape(-1)
        self.index = [torch.from_numpy(np.nonzero(self.which == k)[0]).cuda() for k in range(len(kinds))]
        self.ops = [self._operators(k) for k in kinds]

    @staticmethod
    def _matrix(key, table, wide, centred, skip):
        n = len(key)
        m = np.zeros((n, n))
        for i, k in enumerate(key):
            if k == 9:
                m[i, i] = skip
                continue
            w0 = i - (centred - 1) // 2 if k == 4 else i - k if k < 4 else i + 8 - k - (wide - 1)
            for t in range(centred if k == 4 else wide):
                if 0 <= w0 + t < n:  # halo cells are zero
                    m[i, w0 + t] = table[k, t]
        return torch.from_numpy(m).cuda()

    def _operators(self, key):
        first, second = (self._matrix(key, t, 6, 5, 0.0) for t in (SBP1, SBP2))
        tg = self._matrix(key, TGF, 11, 9, 1.0)
        if self.along_z:  # in place: point i reads the filtered points before it
            low = torch.tril(tg, -1)
            tg = torch.linalg.solve_triangular(torch.eye(len(key), dtype=torch.float64, device="cuda") - low, tg - low,
                                               upper=False)
        return {"first": first.T.contiguous(), "second": second.T.contiguous(),
                "fourth": (second @ second).T.contiguous(), "filter": tg.T.contiguous()}

    def __call__(self, name, f):
        f = f if self.along_z else f.transpose(-1, -2)
        if len(self.ops) == 1:
            out = f @ self.ops[0][name]
        else:
            out = torch.empty(f.shape, dtype=f.dtype, device=f.device)
            for at, op in zip(self.index, self.ops):
                out[..., at, :] = f[..., at, :] @ op[name]
        return out if self.along_z else out.transpose(-1, -2)


class _Flow:
    """The solver's step (right-hand side, RK4, time step) on one block in 64 bits."""

    def __init__(self, f):
        self.p, Nz, Nr = f["params"], f["Nz"], f["Nr"]
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.z, self.r = t(f["z"]), t(f["r"])
        zr, rr = np.full((Nr, Nz), 4), np.full((Nr, Nz), 4)
        self.patches = _patches(f["records"], Nz, Nr)
        for i0, i1, j0, j1, _, d in self.patches:
            if abs(d) == 1:
                i = np.arange(i0, i1 + 1)
                zr[j0:j1 + 1, i0:i1 + 1] = (i - i0 if d == 1 else 8 + i - i1)[None, :]
            else:
                j = np.arange(j0, j1 + 1)
                rr[j0:j1 + 1, i0:i1 + 1] = (j - j0 if d == 2 else 8 + j - j1)[:, None]
        blank = f["ibval"] == 0.0
        self.blank = t(blank)
        self.Z, self.R = _Lines(zr, blank, True), _Lines(rr, blank, False)
        mz, mr = 1.0 / _metric(f["z"]), 1.0 / _metric(f["r"])
        self.mz, self.mr = t(mz)[None, :], t(mr)[:, None]
        self.mz2, self.mr2 = t(_metric(mz))[None, :], t(_metric(mr))[:, None]
        for name, x in (("dz", f["z"]), ("dr", f["r"])):
            d = np.empty(len(x))
            d[1:-1] = (x[2:] - x[:-2]) / 2.0
            d[0], d[-1] = x[1] - x[0], x[-1] - x[-2]
            setattr(self, name, t(d)[None, :] if name == "dz" else t(d)[:, None])
        self.pv, self.target = t(f["pv"]), t(f["target"])
        self.stale = 0.0
        self.time = 0.0

    def dt(self, pv, stale=None):
        """ComputeTimeStep."""
        p, mu = self.p, pv[4] ** 0.666
        s = (pv[4] if p.dt_mode == 1 else torch.full_like(pv[4], self.stale if stale is None else stale)).sqrt()
        inv = (pv[3] * self.mz + pv[1] * self.mr).abs() + s * (self.mz ** 2 + self.mr ** 2).sqrt()
        visc = 2.0 * torch.maximum(mu / p.Re, mu / (p.Re * p.Pr)) * (self.mz.abs() + self.mr.abs()) ** 2
        return float(torch.where(self.blank, 100.0, p.CFL / (inv + visc)).min())

    def sensor(self, pv, dz1, dr1, vr_r):
        """The three artificial coefficients: fourth differences, filters, scaling, ramp."""
        p, rho, T = self.p, pv[0], pv[4]
        dil = dr1[1] + vr_r + dz1[3]
        dil[0] = 2.0 * dr1[1][0] + dz1[3][0]
        s22 = vr_r - dil / 3.0
        s22[0] = dr1[1][0] - dil[0] / 3.0
        s13 = 0.5 * (dz1[1] + dr1[3])
        S = ((dr1[1] - dil / 3.0) ** 2 + 2.0 * s13 ** 2 + s22 ** 2 + (dz1[3] - dil / 3.0) ** 2).sqrt()
        g = torch.stack([S, dil, T])
        z4, r4 = self.Z("fourth", g), self.R("fourth", g)
        vort = dz1[1] - dr1[3]
        fsw = torch.where(-dil < 0.0, 0.0, 1.0) * dil ** 2 / (dil ** 2 + vort ** 2 + float(np.float32(1e-15)))
        q = torch.stack([rho * (z4[0] * self.dz ** 2 + r4[0] * self.dr ** 2).abs(),
                         rho * fsw * (z4[1] * self.dz ** 2 + r4[1] * self.dr ** 2).abs(),
                         rho / (p.gam * T.sqrt()) * (z4[2] * self.dz + r4[2] * self.dr).abs()])
        q = torch.where(self.blank, 0.0, self.R("filter", self.Z("filter", q)))
        ramp = 0.5 * (1.0 + torch.tanh(5.0 * (self.z - 10.0)))[None, :]
        return q[0] * p.C_mu * p.Re * ramp, q[1] * p.C_beta * p.Re * ramp, q[2] * p.C_kappa * p.Re * p.Pr * ramp

    def rhs(self, pv, t):
        p, gam = self.p, self.p.gam
        rho, Vr, Vt, Vz, T = pv
        R = self.r[:, None].clone()
        R[0] = 1.0  # the axis row takes no 1/r term
        six = torch.cat([pv, (rho * T)[None]])
        dz1, dr1 = self.Z("first", six) * self.mz, self.R("first", six) * self.mr
        mu = T ** 0.666
        beta, kap, vr_r = 0.6 * mu, mu.clone(), Vr / R
        if p.shock_capturing == 1:
            ms, bs, ks = self.sensor(pv, dz1, dr1, vr_r)
            mu, beta, kap = mu + ms, beta + bs, kap + ks
        lam = beta - 2.0 / 3.0 * mu
        div = dr1[1] + vr_r + dz1[3]
        conv = Vr * dr1[:5] + Vz * dz1[:5]
        conv[0] += rho * div
        conv[1] += dr1[5] / (gam * rho)
        conv[2] += Vt * vr_r
        conv[3] += dz1[5] / (gam * rho)
        conv[4] += (gam - 1.0) * T * div
        out = -conv
        z2 = self.Z("second", pv[1:]) * self.mz ** 2 + dz1[1:5] * self.mz2
        r2 = self.R("second", pv[1:]) * self.mr ** 2 + dr1[1:5] * self.mr2
        co = torch.stack([mu, kap])
        coz, cor = self.Z("first", co) * self.mz, self.R("first", co) * self.mr
        mix = self.R("first", dz1[[1, 3]]) * self.mr
        q = lam / mu if p.shock_capturing == 1 else torch.full_like(mu, -1.0 / 15.0)
        a, b, m = 2.0 + q, 1.0 + q, -q
        (rz, tz, vz, Tz), (rr, tr, vr, Tr), o = dz1[1:5], dr1[1:5], 1.0 / R
        c = 1.0 / (p.Re * rho)
        normal_r = a * rr - m * vr_r - m * vz
        normal_z = a * vz - m * rr - m * vr_r
        out[1] += c * (mu * (a * r2[0] + a * o * rr + b * mix[1] + z2[0] - a * vr_r * o) + cor[0] * normal_r
                       + coz[0] * (rz + vr))
        out[2] += c * (mu * (r2[1] + z2[1] + o * tr - Vt * o * o) + cor[0] * (tr - Vt * o) + coz[0] * tz)
        out[3] += c * (mu * (r2[2] + a * z2[2] + b * mix[0] + o * vr + b * o * rz) + cor[0] * (vr + rz)
                       + coz[0] * normal_z)
        out[4] += gam / (p.Re * p.Pr * rho) * (kap * (r2[3] + o * Tr + z2[3]) + cor[1] * Tr + coz[1] * Tz)
        out[4] += gam * (gam - 1.0) / p.Re * mu / rho * (
            rr * normal_r + (tr - Vt * o) * (tr - vr_r) + vr_r * (a * vr_r - m * rr - m * vz) + tz * tz
            + vz * normal_z + (rz + vr) ** 2)
        out[:, 0] = 0.0
        if p.control_forcing:
            G = torch.exp(-((self.z[None, :] - p.forcing_z0) / p.forcing_lz) ** 2
                          - ((self.r[:, None] - p.forcing_r0) / p.forcing_lr) ** 2)
            if p.control_forcing == 1:
                F = torch.tensor(list(p.forcing_mat), dtype=torch.float64, device="cuda").reshape(5, 5)
                out += p.forcing_alpha * G * torch.einsum("ek,kji->eji", F, pv - self.target)
            else:
                om = 2.0 * math.pi * p.harmonic_st * p.harmonic_uj
                out[3] += p.harmonic_amp * om * math.cos(om * t) * G
        self.faces(out, pv, dz1, dr1)
        zeta = (self.r - p.sponge_start_top) / (self.r[-1] - p.sponge_start_top)
        zeta = torch.where(self.r >= p.sponge_start_top, zeta, 0.0)
        out -= p.sponge_A_top * (zeta ** 2)[:, None] * (pv - self.target)
        zeta = ((p.sponge_end_left - self.z) / p.sponge_end_left).clamp(min=0.0)
        out[:, 1:] -= p.sponge_A_left * (zeta ** 2)[None, :] * (pv - self.target)[:, 1:]
        return out

    def faces(self, out, pv, dz1, dr1):
        """SAT and NSCBC closures, patch by patch."""
        gam, g1 = self.p.gam, self.p.gam - 1.0
        for i0, i1, j0, j1, bc, d in self.patches:
            if bc == 90 or (bc == 91 and abs(d) == 2):
                continue
            if bc in (91, 92):
                j0 = max(j0, 1)
            at = {1: (slice(j0, j1 + 1), slice(i0, i0 + 1)), -1: (slice(j0, j1 + 1), slice(i1, i1 + 1)),
                  2: (slice(j0, j0 + 1), slice(i0, i1 + 1)), -2: (slice(j1, j1 + 1), slice(i0, i1 + 1))}[d]
            at = (slice(None),) + at
            u, tgt, o, gz, gr = pv[at], self.target[at], out[at], dz1[at], dr1[at]
            rho, Vr, Vt, Vz, T = u
            along, n = (Vz, 3) if abs(d) == 1 else (Vr, 1)
            met = (self.mz.expand(pv.shape[1:]) if abs(d) == 1 else self.mr.expand(pv.shape[1:]))[at[1:]]
            sT = T.sqrt()
            lam = torch.stack([along, along, along, along - sT, along + sT])

            def to_waves(v):
                # entropy, the two shears, and the two acoustic waves along the face's normal
                ent = -g1 * T / (gam * rho) * v[0] + v[4] / gam
                ac = g1 * T / (2.0 * gam * rho) * v[0] + g1 / (2.0 * gam) * v[4]
                return torch.stack([ent, v[2], v[1] if n == 3 else v[3], ac - 0.5 * g1 * sT * v[n],
                                    ac + 0.5 * g1 * sT * v[n]])

            def from_waves(w):
                tp = rho / (g1 * T)
                res = torch.empty_like(w)
                res[0] = -rho / T * w[0] + tp * (w[3] + w[4])
                res[2] = w[1]
                res[1 if n == 3 else 3] = w[2]
                res[n] = (w[4] - w[3]) / (g1 * sT)
                res[4] = w[0] + w[3] + w[4]
                return res

            if bc in (91, 93):
                lin = (lam.abs() + lam) / 2.0 if d > 0 else (lam.abs() - lam) / 2.0
                ref = tgt
                if bc == 93:
                    ref = u.clone()
                    ref[n] = 0.0
                o += -2.0 * met * 48.0 / 49.0 * from_waves(lin * to_waves(u - ref))
                if bc == 93:
                    wall = u.clone()
                    wall[1:4] = 0.0
                    wall[4] = tgt[4]
                    o += -2.0 * met * 48.0 / 49.0 * (u - wall)
                continue
            gn = gz if abs(d) == 1 else gr
            if bc == 92:
                add = along * gn[:5]
                add[0] += rho * gn[n]
                add[n] += gn[5] / (gam * rho)
                add[4] += g1 * T * gn[n]
                w = to_waves(gz[:5])  # z derivatives on r faces as well
                w = torch.where((lam > 0.0) if d > 0 else (lam < 0.0), 0.0, w)
                o += add - from_waves(lam * w)
            else:
                w = to_waves(gn[:5])
                if d < 0:
                    w[3] = -w[4]
                else:
                    w[4] = -w[3]
                o[0] += along * gn[0] + rho * gn[n]
                o -= from_waves(lam * w)
                o[1:] = 0.0

    def axis(self, pv, src):
        s = torch.from_numpy(SBP1[0, 1:]).cuda()
        for e in (0, 3, 4):
            pv[e, 0] = -(s[:, None] * src[e, 1:6]).sum(0) / SBP1[0, 0]

    def step(self, dt):
        """RK4: the axis closure follows each stage with the stage input's values."""
        old, cur, ks = self.pv, self.pv, []
        for a, ct in ((0.5, 0.0), (0.5, 0.5), (1.0, 0.5), (None, 1.0)):
            k = dt * self.rhs(cur, self.time + ct * dt)
            ks.append(k)
            if a is None:
                break
            nxt = old + a * k
            self.axis(nxt, cur)
            cur = nxt
        new = old + ks[0] / 6.0 + (ks[1] + ks[2]) / 3.0 + ks[3] / 6.0
        new = torch.where(self.blank, cur, new)
        self.axis(new, cur)
        self.stale = float(cur[4, -1, -1])  # the temperature at the last face point
        self.pv, self.time = new, self.time + dt


def _advanced(f, steps):
    flow = _Flow(f)
    for _ in range(steps):
        dt = flow.dt(flow.pv)
        flow.step(dt)
    return flow.pv, dt


def exact(case, seed):
    c = _full(case)
    if c["kind"] == "train" or c["sensor"]:
        # the network's draws and the judge's held values have no value in 64 bits
        return None
    if c["kind"] == "dt":
        f = _dt_fixture(c, seed)
        flow = _Flow.__new__(_Flow)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        flow.p, flow.blank = f["params"], torch.zeros((c["Nr"], c["Nz"]), dtype=torch.bool, device="cuda")
        flow.mz, flow.mr = t(1.0 / _metric(f["z"]))[None, :], t(1.0 / _metric(f["r"]))[:, None]
        return torch.tensor([flow.dt(t(f["pv"]), stale=1.0)], dtype=torch.float64)
    if c["kind"] == "batch":
        return [_advanced(f, c["steps"])[0] for f in _batch_fixtures(case, seed)]
    pv, dt = _advanced(_fixture(case, seed), c["steps"])
    return {"pv": pv, "dt": dt}
