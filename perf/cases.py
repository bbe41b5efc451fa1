"""The work that a user of this framework has it do, as cases that can be timed.

Each case is one pass through the public entry points (cuda_sto_pf_gb300's
Solver, WarmStartModel and the C ABI that they wrap).  The kinds:

dynamics   fields loaded, `steps` time steps, fields read back: what
           main_cuda --mode=dynamics and a Python driver do
minimize   fields loaded, `steps` minimize iterations, fields read back
sweep      pfgb_batch_minimize over several uneven grids, host fields in and out
fft        one 3D transform of the library's own (r2c, c2r, r2c_noalloc)
fno        the learned elastic start: one forward
fno_train  the same model: gradients over a few pairs and one Adam step

exact() restates dynamics, minimize, the transforms and the model in float64
torch.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

from cuda_sto_pf_gb300 import capi
from cuda_sto_pf_gb300.fno import WarmStartModel
from cuda_sto_pf_gb300.solver import Solver

PARAMS = os.path.join("tests", "golden", "c2.params")
XB_MAX_SAFE = 0.07            # the raw-field loader's default cap
IFACE_W = 2.5                 # ic_phi_iface_w of PARAMS
EIGEN_DIAG = (0.046, -0.022, -0.017)
GP_X, GP_DG0 = 0.3529411764705882, 0.0
RGAS = 8.31446261815324
F64, C128 = torch.float64, torch.complex128


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _dyn(name, nx, ny, nz, steps, prec, model, elastic="hetero", zero_mode=True, solver="default",
         y_mode="lagged", diag=False):
    return {"name": name, "kind": "dynamics", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "prec": prec,
            "model": model, "elastic": elastic, "zero_mode": zero_mode, "solver": solver, "y_mode": y_mode,
            "diag": diag}


def listed():
    return [
        # a small grid's forward transform by a caller that cannot allocate:
        # launches and latency
        {"name": "fft_noalloc_fp32_24", "kind": "fft", "op": "r2c_noalloc", "prec": "fp32", "nx": 24, "ny": 24,
         "nz": 24},
        # a ragged grid's inverse transform in FP64 (the input is workspace,
        # so a caller that keeps its spectrum copies it first)
        {"name": "fft_c2r_fp64_90x75x126", "kind": "fft", "op": "c2r", "prec": "fp64", "nx": 90, "ny": 75, "nz": 126},
        # the flagship grid's forward transform
        {"name": "fft_r2c_fp32_246", "kind": "fft", "op": "r2c", "prec": "fp32", "nx": 246, "ny": 246, "nz": 246},
        # the plain method: one sphere, homogeneous elasticity, FP64, a CSV
        # row (diagnostics) at every step
        _dyn("dyn_fp64_64_homogeneous", 64, 64, 64, 10, "fp64", "two_phase", elastic="homogeneous", diag=True),
        # the CLI's default precision on a mid-size grid
        _dyn("dyn_fp64_128_gp", 128, 128, 128, 4, "fp64", "gp_zone", zero_mode=False),
        # the reference's default elastic solver on an uneven grid, FP32
        _dyn("dyn_fp32_104x90x135", 104, 90, 135, 5, "fp32", "two_phase"),
        # the headline run: 246^3, GP zone, heterogeneous elasticity to 1e-8
        # with the Chebyshev update and the extrapolated start
        _dyn("dyn_fp32_246_gp", 246, 246, 246, 10, "fp32", "gp_zone", solver="accelerated"),
        # the largest grid: one cold step
        _dyn("dyn_fp32_512_gp", 512, 512, 512, 1, "fp32", "gp_zone", solver="accelerated"),
        # one case of the minimize sweep
        {"name": "min_fp32_96", "kind": "minimize", "n": 96, "steps": 10, "prec": "fp32", "aspect": 0.6},
        # the batched sweep over uneven grids
        {"name": "sweep_fp32_64_to_144", "kind": "sweep", "sizes": "64,80,96,112,128,144", "steps": 8,
         "concurrency": 6},
        # the learned start: a prediction and a training step
        {"name": "fno_forward_128", "kind": "fno", "n": 128, "modes": 12, "layers": 4},
        {"name": "fno_train_64", "kind": "fno_train", "n": 64, "modes": 8, "layers": 4, "pairs": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["dynamics", "minimize", "sweep", "fft", "fno", "fno_train"], [9, 3, 1, 4, 2, 2])[0]
    if kind == "dynamics":
        while True:
            nx, ny, nz = (_log_int(rng, 24, 288) for _ in range(3))
            if 24 ** 3 <= nx * ny * nz <= 9_000_000:
                break
        model = rng.choice(["two_phase", "gp_zone"])
        y_mode = "x_split" if model == "two_phase" and rng.random() < 0.15 else "lagged"
        c = _dyn("", nx, ny, nz, rng.randint(1, 6), rng.choice(["fp32", "fp32", "fp64"]), model,
                 elastic=rng.choices(["hetero", "homogeneous", "off"], [6, 2, 1])[0],
                 zero_mode=y_mode == "lagged" and rng.random() < 0.6,
                 solver=rng.choice(["default", "accelerated"]), y_mode=y_mode, diag=rng.random() < 0.3)
        del c["name"]
        return c
    if kind == "minimize":
        return {"kind": kind, "n": _log_int(rng, 48, 168), "steps": rng.randint(2, 10),
                "prec": rng.choice(["fp32", "fp64"]), "aspect": rng.choice([1.0, 0.6, 0.3])}
    if kind == "sweep":
        sizes = [16 * rng.randint(4, 9) for _ in range(rng.randint(2, 6))]
        return {"kind": kind, "sizes": ",".join(str(s) for s in sizes), "steps": rng.randint(3, 8),
                "concurrency": rng.randint(2, 8)}
    if kind == "fft":
        while True:
            nx, ny, nz = (_log_int(rng, 20, 400) for _ in range(3))
            if nx * ny * nz <= 20_000_000:
                break
        return {"kind": kind, "op": rng.choice(["r2c", "c2r", "r2c_noalloc"]), "prec": rng.choice(["fp32", "fp64"]),
                "nx": nx, "ny": ny, "nz": nz}
    n = _log_int(rng, 32, 128 if kind == "fno" else 80)
    m = rng.randint(4, min(12, n // 4))
    c = {"kind": kind, "n": n, "modes": m, "layers": rng.choice([2, 4])}
    if kind == "fno_train":
        c["pairs"] = rng.randint(1, 3)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _axis_box(c, half, n):
    lo, hi = math.floor(c - half), math.ceil(c + half)
    return np.arange(n) if hi - lo + 1 >= n else np.arange(lo, hi + 1) % n


def _add_ellipsoid(field, centre, radii, rot):
    """field <- max(field, the tanh seed profile of one ellipsoid), periodic"""
    shape, dev = field.shape, field.device
    half = max(radii) + 8.0 * IFACE_W
    idx = [torch.from_numpy(_axis_box(c, half, n)).to(dev) for c, n in zip(centre, shape)]
    d = []
    for a, n in enumerate(shape):
        x = idx[a].to(F64) - float(centre[a])
        d.append(x - n * torch.round(x / n))
    r2 = 0.0
    for a in range(3):
        q = (rot[a][0] * d[0])[:, None, None] + (rot[a][1] * d[1])[None, :, None] + (rot[a][2] * d[2])[None, None, :]
        r2 = r2 + (q / radii[a]) ** 2
    seed = 0.5 * (1.0 + torch.tanh((1.0 - torch.sqrt(r2)) * (min(radii) / IFACE_W)))
    at = (idx[0][:, None, None], idx[1][None, :, None], idx[2][None, None, :])
    field[at] = torch.maximum(field[at], seed)


def _rotation(rng):
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    return [[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
            [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
            [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]]


def _composition(phi, seed):
    """0.03 + N(0, 1e-3) in the matrix, 0.33 in precipitates, under the loader's cap"""
    g = torch.Generator(device=phi.device)
    g.manual_seed(int(seed))
    h = phi ** 3 * (6 * phi ** 2 - 15 * phi + 10)
    base = 0.03 + 1e-3 * torch.randn(phi.shape, dtype=F64, device=phi.device, generator=g)
    return ((1 - h) * base + h * 0.33).clamp(1e-8, XB_MAX_SAFE)


def _population(shape, seed):
    """non-overlapping ellipsoids (log-normal radii, random rotations) and
    GP-zone eta sites, in the headline run's density"""
    rng = np.random.default_rng(seed)
    L = np.array(shape, dtype=float)
    frac = float(np.prod(L)) / 246.0 ** 3
    count, sites = max(1, round(60 * frac)), max(1, round(20 * frac))
    cs, rs, rots = [], [], []
    for _ in range(400 * count):
        if len(cs) >= count:
            break
        a = 6.0 * math.exp(0.3 * rng.standard_normal())
        R = np.array([a, a * rng.uniform(0.5, 1.0), a * rng.uniform(0.5, 1.0)])
        c = rng.uniform(size=3) * L
        if cs:
            d = np.array(cs) - c
            d -= L * np.round(d / L)
            if np.any(np.linalg.norm(d, axis=1) < np.array([r.max() for r in rs]) + R.max() + 2 * IFACE_W):
                continue
        cs.append(c), rs.append(R), rots.append(_rotation(rng))
    phi = torch.zeros(shape, dtype=F64, device="cuda")
    eta = torch.zeros(shape, dtype=F64, device="cuda")
    for c, R, M in zip(cs, rs, rots):
        _add_ellipsoid(phi, c, R, M)
    for _ in range(sites):
        _add_ellipsoid(eta, rng.uniform(size=3) * L, np.full(3, 3.0), np.eye(3).tolist())
    return phi, _composition(phi, seed), eta * (1.0 - phi).clamp(0, 1)


def _spheroid(n, aspect, seed):
    """a centred spheroid seed, the rotation it shares with its eigenstrain,
    and the eigenstrain (xx, yy, zz, yz, xz, xy)"""
    rng = np.random.default_rng(seed)
    R = min(rng.uniform(10.0, 40.0), n / 2 - 2 * IFACE_W - 1)
    M = _rotation(rng)
    phi = torch.zeros((n, n, n), dtype=F64, device="cuda")
    _add_ellipsoid(phi, np.full(3, n / 2), np.array([R, R, aspect * R]), M)
    A = np.array(M)
    E = A @ np.diag(EIGEN_DIAG) @ A.T
    return phi, _composition(phi, seed), [E[0, 0], E[1, 1], E[2, 2], E[1, 2], E[0, 2], E[0, 1]]


def _fields(case, seed):
    if case["kind"] == "minimize":
        return _spheroid(case["n"], case["aspect"], seed)
    shape = (case["nx"], case["ny"], case["nz"])
    if case["elastic"] == "homogeneous" and case["model"] == "two_phase":   # one centred sphere
        rng = np.random.default_rng(seed)
        phi = torch.zeros(shape, dtype=F64, device="cuda")
        _add_ellipsoid(phi, np.array(shape) / 2 + rng.uniform(-2, 2, 3), np.full(3, 8.0), np.eye(3).tolist())
        return phi, _composition(phi, seed), torch.zeros(shape, dtype=F64, device="cuda")
    return _population(shape, seed)


def _params(case):
    p = capi.load_params_file(PARAMS)
    p.precision = capi.PREC_FP32 if case.get("prec", "fp32") == "fp32" else capi.PREC_FP64
    if case["kind"] == "dynamics":
        p.Nx, p.Ny, p.Nz = case["nx"], case["ny"], case["nz"]
        p.model_mode = capi.MODEL_GP_ZONE if case["model"] == "gp_zone" else capi.MODEL_TWO_PHASE
        p.zero_mode_enabled = 1 if case["zero_mode"] else 0
        p.elastic_fail_on_nonconvergence = 0
        if case["elastic"] == "off":
            p.elastic_enabled = 0
        if case["elastic"] == "homogeneous":
            for i in range(21):
                p.S_p[i] = 0.0
        if case["solver"] == "accelerated":
            p.elastic_residual_tolerance = 1e-8
            p.elastic_chebyshev = 1
            p.elastic_warm_start_extrapolate = 5
        if case["y_mode"] == "x_split":
            capi.set_param(p, "pf_y_update_mode", "x_transport_projection_split")
    else:
        p.Nx = p.Ny = p.Nz = case["n"]
        p.mode = capi.MODE_MINIMIZE
        p.minimize_full_model = 1
        p.minimize_dt = 0.05
        p.minimize_V0 = 0.1
    return p


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _pinned(shape):
    return torch.empty(shape, dtype=F64, pin_memory=True)


def _real(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    dt = torch.float32 if case["prec"] == "fp32" else F64
    return torch.randn((case["nx"], case["ny"], case["nz"]), dtype=dt, device="cuda", generator=g)


def _fno_layout(case):
    m = 4 * case["modes"] ** 3
    out = [("P", (32, 8)), ("p", (32,))]
    for i in range(case["layers"]):
        out += [("W%d" % i, (32, 32)), ("b%d" % i, (32,)), ("R%d" % i, (32, 32, m, 2))]
    return out + [("Q1", (64, 32)), ("q1", (64,)), ("Q2", (3, 64)), ("q2", (3,))]


def _fno_weights(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    blocks = {}
    for name, shape in _fno_layout(case):
        scale = 0.1 if len(shape) == 1 else 1 / 32 if name[0] == "R" else 1 / math.sqrt(shape[1])
        blocks[name] = scale * torch.randn(shape, dtype=torch.float32, device="cuda", generator=g)
    return blocks


FNO_IN = (2.0, 4.0, 60.0, 60.0, 60.0, 30.0, 30.0, 30.0)
FNO_OUT = (0.05, 0.04, 0.03)


def _fno_pair(case, seed):
    """the model's eight inputs (phi, eta, eigenstrain) and a smooth target"""
    n = case["n"]
    phi, xB, eta = _population((n, n, n), seed)
    h = phi ** 3 * (6 * phi ** 2 - 15 * phi + 10)
    rng = np.random.default_rng(seed)
    A = np.array(_rotation(rng))
    E = A @ np.diag(EIGEN_DIAG) @ A.T
    e = [(1 - h) * xB * 2.33e-3 + h * E[a, a] for a in range(3)] + [h * E[1, 2], h * E[0, 2], h * E[0, 1]]
    x = torch.stack([phi, eta] + e).float().contiguous()
    t = torch.zeros((3, n, n, n), dtype=F64, device="cuda")
    r = torch.arange(n, dtype=F64, device="cuda") * (2 * math.pi / n)
    for c in range(3):
        for _ in range(6):
            k = rng.integers(-3, 4, 3)
            ph = (k[0] * r)[:, None, None] + (k[1] * r)[None, :, None] + (k[2] * r)[None, None, :]
            t[c] += FNO_OUT[c] * rng.normal() * torch.cos(ph + rng.uniform(0, 2 * math.pi))
    return x, t.float().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "fft":
        x = _real(case, seed)
        nzc = case["nz"] // 2 + 1
        ct = torch.complex64 if case["prec"] == "fp32" else C128
        if case["op"] == "c2r":
            st["spec"] = torch.fft.rfftn(x).contiguous()
            st["work"] = torch.empty_like(st["spec"])
            st["out"] = torch.empty_like(x)
        else:
            st["x"] = x
            st["out"] = torch.empty((case["nx"], case["ny"], nzc), dtype=ct, device="cuda")
        st["lib"] = capi.load()
        return st
    if kind in ("dynamics", "minimize"):
        f = _fields(case, seed)
        p = _params(case)
        if kind == "minimize":
            for i in range(6):
                p.eps00[i] = f[2][i]
        capi.finalize(p)
        st["solver"] = Solver(p)
        st["solver"].set_stream(torch.cuda.current_stream().cuda_stream)
        st["phi"], st["xB"] = f[0], f[1]
        st["eta"] = f[2] if kind == "dynamics" and case["model"] == "gp_zone" else None
        st["out"] = {k: _pinned(f[0].shape) for k in ("phi", "xB") + (("eta",) if st["eta"] is not None else ())}
        return st
    if kind == "sweep":
        sizes = [int(s) for s in case["sizes"].split(",")]
        arr, keep = (capi.Case * len(sizes))(), []
        for i, n in enumerate(sizes):
            c = {"kind": "minimize", "n": n, "prec": "fp32", "aspect": (1.0, 0.6, 0.3)[i % 3]}
            phi, xB, e00 = _spheroid(n, c["aspect"], seed + 1000 * i)
            p = _params(c)
            for k in range(6):
                p.eps00[k] = e00[k]
            capi.finalize(p)
            bufs = [phi.cpu().numpy(), xB.cpu().numpy(), np.zeros(phi.shape), np.zeros(phi.shape)]
            keep.append(bufs)
            arr[i].params = p
            arr[i].phi, arr[i].xB, arr[i].phi_out, arr[i].xB_out = (b.ctypes.data for b in bufs)
            arr[i].max_iter = case["steps"]
            arr[i].stop_on_convergence = 0
        st.update(arr=arr, keep=keep, lib=capi.load())
        return st
    n = case["n"]
    m = WarmStartModel((n, n, n), modes=case["modes"], layers=case["layers"], in_scale=FNO_IN, out_scale=FNO_OUT)
    w = _fno_weights(case, seed)
    m.set_params(torch.cat([w[k].reshape(-1) for k, _ in _fno_layout(case)]).cpu().numpy())
    m.set_stream(torch.cuda.current_stream().cuda_stream)
    st["model"] = m
    st["pairs"] = [_fno_pair(case, seed + 77 * i) for i in range(case.get("pairs", 1))]
    if kind == "fno":
        st["out"] = torch.empty((3, n, n, n), dtype=torch.float32, device="cuda")
    else:
        st["grad"] = torch.empty(m.num_params, dtype=torch.float32, pin_memory=True)
    return st


def _take(buf, case):
    """A result at the precision that the run carries, which goes on to the
    device: float32 for FP32 fields, and with elasticity, whose strain is
    single precision in every run (as in the reference), for FP64 fields too;
    FP64 fields without elasticity stay float64."""
    if case["prec"] == "fp64" and case.get("elastic") == "off":
        return buf
    return buf.to("cuda", non_blocking=True).float()


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "fft":
        lib, out = st["lib"], st["out"]
        if case["op"] == "c2r":
            st["work"].copy_(st["spec"])
            src, fn = st["work"], lib.pfgb_fft3d_c2r
        else:
            src = st["x"]
            fn = lib.pfgb_fft3d_r2c if case["op"] == "r2c" else lib.pfgb_fft3d_r2c_noalloc
        capi.check(fn(capi.PREC_FP32 if case["prec"] == "fp32" else capi.PREC_FP64, case["nx"], case["ny"], case["nz"],
                      src.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream), case["op"])
        return out
    if kind in ("dynamics", "minimize"):
        s, out = st["solver"], st["out"]
        s.load_device(st["phi"], st["xB"], st["eta"])
        extra = {}
        if kind == "minimize":
            m = s.minimize(case["steps"])
            extra = {"mean_h": m.mean_h, "F_surf": m.F_surf, "F_el": m.F_el}
        elif case["diag"]:
            rows = []
            for _ in range(case["steps"]):
                s.step(1)
                d = s.diagnostics()
                rows.append([d.vf_precip, d.mass_xBtot / s.N, d.mean_xB])
            extra = {"rows": torch.tensor(rows, dtype=torch.float32)}
        else:
            s.step(case["steps"])
        s.read_into(**out)
        return {**{k: _take(v, case) for k, v in out.items()}, **extra}
    if kind == "sweep":
        arr = st["arr"]
        capi.check(st["lib"].pfgb_batch_minimize(arr, len(arr), 0, case["concurrency"]), "sweep")
        return [[b.astype(np.float32) for b in bufs[2:]] for bufs in st["keep"]]
    m = st["model"]
    if kind == "fno":
        m.forward(st["pairs"][0][0], st["out"])
        return st["out"]
    losses = [m.loss_grad(x, t, accumulate=i > 0) for i, (x, t) in enumerate(st["pairs"])]
    capi.check(m.lib.pfgb_fno_get_grad(m.handle, st["grad"].data_ptr(), st["grad"].numel()), "get_grad")
    m.adam_step(1e-4, clip_norm=1.0)
    return {"grad": st["grad"], "loss": losses}


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------
def _cells(case):
    return case["n"] ** 3 if "n" in case else case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Inputs read once and outputs written once; a time step or iteration
    also has to read and write its state once.  The elastic iteration counts
    its two real transforms of six fields per update, four updates a step."""
    kind = case["kind"]
    if kind == "sweep":
        w = [work({"kind": "minimize", "n": int(s), "steps": case["steps"], "prec": "fp32"})
             for s in case["sizes"].split(",")]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    n = _cells(case)
    fft = 2.5 * n * math.log2(n)     # one real transform
    size = 4 if case.get("prec", "fp32") == "fp32" else 8
    if kind == "fft":
        return {"bytes": 2.0 * n * size, "flops": fft}
    if kind in ("dynamics", "minimize"):
        fields = 3 if case.get("model") == "gp_zone" else 2
        state = 2.0 * n * ((fields + 1) * size + (0 if case.get("elastic") == "off" else 12))
        transforms = (14 if kind == "minimize" else 8 + 2 * fields) + (0 if case.get("elastic") == "off" else 48)
        return {"bytes": 2.0 * n * 8 * fields + case["steps"] * state, "flops": case["steps"] * transforms * fft}
    m, L = 2 * case["modes"], case["layers"]
    weights = 2.0 * 32 * 32 * L * (m * m * m / 2) * 2
    flops = 2.0 * n * (8 * 32 + L * 32 * 32 + 32 * 64 + 64 * 3) + L * 2 * 32 * fft
    if kind == "fno":
        return {"bytes": 4.0 * 11 * n + weights, "flops": flops}
    return {"bytes": case["pairs"] * (4.0 * 11 * n + weights) + 6 * weights, "flops": 3.0 * case["pairs"] * flops}


# ---------------------------------------------------------------------------
# the same in float64
# ---------------------------------------------------------------------------
def _h(p):
    return p ** 3 * (6 * p * p - 15 * p + 10)


def _hp(p):
    return 30 * p * p * (1 - p) ** 2


class _Model:
    """The phase-field model of PARAMS on one grid, in float64 torch."""

    def __init__(self, shape, prm, hetero=True, eps00=None, dt=None):
        self.q = prm
        self.shape, self.dev = shape, "cuda"
        self.N = shape[0] * shape[1] * shape[2]
        self.dt = prm["dt"] if dt is None else dt
        ks, ms = [], []
        for a, n in enumerate(shape):
            i = torch.arange(n if a < 2 else n // 2 + 1, device=self.dev)
            k = 2 * math.pi * torch.where(i <= n // 2, i, i - n).to(F64) / n
            v = [1, 1, 1]
            v[a] = -1
            ks.append(k.reshape(v))
            ms.append((k.abs() < math.pi * (2.0 / 3.0)).reshape(v))
        self.k = ks
        self.mask = ms[0] & ms[1] & ms[2]
        self.k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
        voigt = {}
        for pre in ("S_", "S_p_"):
            C = np.zeros((6, 6))
            for a in range(6):
                for b in range(a, 6):
                    C[a, b] = C[b, a] = prm["%s%d%d" % (pre, a + 1, b + 1)]
            voigt[pre] = C
        self.C0 = voigt["S_"]
        self.dC = voigt["S_p_"] if hetero else np.zeros((6, 6))
        self.e00 = [prm["eps_%s00" % s] for s in ("xx", "yy", "zz", "yz", "xz", "xy")] if eps00 is None else eps00
        # SGTE unary energies at the run's temperature and the regular solution
        T = prm["temperature_C"] + 273.15
        lnT = T * math.log(T)
        if T < 600.61:
            gpb = -7650.085 + 101.700244 * T - 24.5242231 * lnT - 0.00365895 * T ** 2 - 2.4395e-7 * T ** 3
        else:
            gpb = -10531.095 + 154.243182 * T - 32.4913959 * lnT + 0.00154613 * T ** 2 + 8.05448e25 * T ** -9
        gag = -7209.512 + 118.202013 * T - 23.8463314 * lnT - 0.001790585 * T ** 2 - 3.98587e-7 * T ** 3 - 12011.0 / T
        gte = -10544.679 + 183.372894 * T - 35.6687 * lnT + 0.01583435 * T ** 2 - 5.240417e-6 * T ** 3 + 155015.0 / T
        s = prm["mu_reference_scale"]
        RT, L = RGAS * T, 41212.9 - 18.05 * T
        self.GA = (-76063.2138 + 9.67716633 * T + gpb + gte) / s
        self.GB = 3 * (-10128.93 - 12.645115 * T + 2 / 3 * gag + 1 / 3 * gte) / s
        self.RT, self.L = RT / s, L / s
        x = max(math.exp(-L / RT), 1e-9)      # solubility limit, to the framework's 1e-8
        for _ in range(20):
            d = (RT * math.log(x) + L * (1 - x) ** 2) / (RT / x - 2 * L * (1 - x))
            x = min(max(x - d, 1e-10), 0.999)
            if abs(d) < 1e-8:
                break
        muA, muB = (v + g for v, g in zip(self.off_f(x), (self.GA, self.GB)))
        vA, vB = prm["v_A"], prm["v_B"]
        self.mu0 = (vA * muA + vB * muB) / (vA + vB)
        oA, oB = self.off_f(GP_X)
        self.gpC = oA * (1 - GP_X) + oB * GP_X - GP_DG0
        self.u = None

    def off_f(self, x):
        return self.RT * math.log(1 - x) + self.L * x * x, self.RT * math.log(x) + self.L * (1 - x) ** 2

    def off(self, x):
        x = x.clamp(1e-12, 1 - 1e-12)
        return self.RT * torch.log1p(-x) + self.L * x * x, self.RT * torch.log(x) + self.L * (1 - x) ** 2

    def fwd(self, f):
        return torch.fft.rfftn(f)

    def inv(self, f):
        return torch.fft.irfftn(f, s=self.shape)

    def eigen(self, phi, xB):
        h = _h(phi)
        ea = (1 - h) * (xB.clamp(0, 1) * self.q["eps_iso_over_vB"])
        return [ea + h * self.e00[a] if a < 3 else h * self.e00[a] for a in range(6)]

    def hooke(self, C, e):
        """C : e with engineering shear; zero entries of C skipped"""
        out = []
        for a in range(6):
            acc = None
            for b in range(6):
                c = C[a, b] * (2.0 if b >= 3 else 1.0)
                if c != 0.0:
                    acc = c * e[b] if acc is None else acc + c * e[b]
            out.append(torch.zeros_like(e[0]) if acc is None else acc)
        return out

    def strain_k(self, u):
        k = self.k
        e = [1j * k[a] * u[a] for a in range(3)]
        return e + [0.5j * (k[a] * u[b] + k[b] * u[a]) for a, b in ((1, 2), (0, 2), (0, 1))]

    def green(self, tau):
        k, C = self.k, self.C0
        kf = [v.expand(self.mask.shape) for v in k]
        vi = ((0, 5, 4), (5, 1, 3), (4, 3, 2))
        t = [sum(k[j] * tau[vi[i][j]] for j in range(3)) for i in range(3)]
        K = [[sum((kf[a] * kf[b] * C[vi[i][a], vi[j][b]] for a in range(3) for b in range(3)
                   if C[vi[i][a], vi[j][b]] != 0.0), torch.zeros_like(kf[0])) for j in range(3)] for i in range(3)]
        c00 = K[1][1] * K[2][2] - K[1][2] ** 2
        c01 = K[0][2] * K[1][2] - K[0][1] * K[2][2]
        c02 = K[0][1] * K[1][2] - K[0][2] * K[1][1]
        c11 = K[0][0] * K[2][2] - K[0][2] ** 2
        c12 = K[0][2] * K[0][1] - K[0][0] * K[1][2]
        c22 = K[0][0] * K[1][1] - K[0][1] ** 2
        det = K[0][0] * c00 + K[0][1] * c01 + K[0][2] * c02
        keep = self.mask.clone()
        keep[0, 0, 0] = False
        w = torch.where(keep, 1.0 / torch.where(keep, det, torch.ones_like(det)), torch.zeros_like(det))
        G = ((c00, c01, c02), (c01, c11, c12), (c02, c12, c22))
        return [-1j * (w * (G[i][0] * t[0] + G[i][1] * t[1] + G[i][2] * t[2])) for i in range(3)]

    def elastic(self, phi, xB):
        """the converged strain of the heterogeneous fixed point"""
        e0, h = self.eigen(phi, xB), _h(phi)
        if self.u is None:
            self.u = self.green([self.fwd(v) for v in self.hooke(self.C0, e0)])
        if not self.dC.any():
            self.u = self.green([self.fwd(v) for v in self.hooke(self.C0, e0)])
            return [self.inv(v) for v in self.strain_k(self.u)], e0, h
        w = torch.full((self.shape[2] // 2 + 1,), 2.0, dtype=F64, device=self.dev)
        w[0] = 1.0
        for _ in range(80):
            e = [self.inv(v) for v in self.strain_k(self.u)]
            el = [a - b for a, b in zip(e, e0)]
            t = [a - b - h * c for a, b, c in zip(self.hooke(self.C0, e), self.hooke(self.C0, el),
                                                  self.hooke(self.dC, el))]
            un = self.green([self.fwd(v) for v in t])
            num = sum(float((w * (a - b).abs() ** 2).sum()) for a, b in zip(un, self.u))
            den = sum(float((w * a.abs() ** 2).sum()) for a in un)
            self.u = un
            if num <= 1e-22 * den:
                break
        return [self.inv(v) for v in self.strain_k(self.u)], e0, h

    def stress(self, el, h):
        return [a + h * b for a, b in zip(self.hooke(self.C0, el), self.hooke(self.dC, el))]

    def phi_rhs(self, phi, xB, el, sig):
        q, h, hp = self.q, _h(phi), _hp(phi)
        f = q["W"] * 2 * phi * (1 - phi) * (1 - 2 * phi)
        x = xB.clamp(0, 1)
        oA, oB = self.off(x)
        Vm0, Vmc, vA, vB, dVm = q["Vm_alpha_0"], q["Vm_compound"], q["v_A"], q["v_B"], q["dVm_alpha_dxB"]
        dmu = self.mu0 - vA * (self.GA + oA) - vB * (self.GB + oB) - (q["elastic_shift_dimless"] if el else 0.0)
        cb = 1.0 / ((Vm0 + dVm * x) * (1 - h) + Vmc * h)
        mt = (1 - h) * ((self.GA + oA) * (1 - x) + (self.GB + oB) * x) + h * self.mu0
        f = f + cb * hp * (dmu - cb * mt * (Vmc - (Vm0 + dVm * x) + dVm * (x - vB)))
        if el:
            eiv = q["eps_iso_over_vB"]
            diag = -x * eiv + eiv * (x - vB)
            de = [hp * (self.e00[a] + diag) if a < 3 else hp * self.e00[a] for a in range(6)]
            Q = sum((2.0 if a >= 3 else 1.0) * v * w for a, (v, w) in enumerate(zip(self.hooke(self.dC, el), el)))
            f = f - sum((2.0 if a >= 3 else 1.0) * sig[a] * de[a] for a in range(6)) + 0.5 * hp * Q
        return f

    def allen_cahn(self, f, Ldt, kappa):
        return self.inv(self.mask * self.fwd(f) / (1 + Ldt * kappa * self.k2))

    def eta_rhs(self, eta, phi, xB):
        q, e, p = self.q, eta.clamp(0, 1), phi.clamp(0, 1)
        x = xB.clamp(1e-12, 1 - 1e-12)
        oA, oB = self.off(x)
        dgg = (self.GB - self.GA) * (GP_X - x) + self.gpC - (oA * (1 - x) + oB * x)
        cref = 1.0 / (q["Vm_alpha_0"] + q["dVm_alpha_dxB"] * x)
        return cref * (1 - _h(p)) * _hp(e) * dgg + q["gp_W_eta_code"] * 2 * e * (1 - e) * (1 - 2 * e)

    def y_update(self, Y, dYdt, pn, pp, eta, sig, gp, zm):
        q, dt, vB = self.q, self.dt, self.q["v_B"]
        phiY = pn if zm else pp
        xc = torch.sigmoid(Y.clamp(-20, 20)).clamp(1e-8, 1 - 1e-8)
        oA, oB = self.off(xc)
        h = _h(phiY)
        Vm = q["Vm_alpha_0"] + q["dVm_alpha_dxB"] * xc
        dG = self.GB - self.GA + oB - oA
        cb = 1.0 / (Vm * (1 - h) + q["Vm_compound"] * h)
        if gp:
            mu = dG / Vm
        else:
            mt = (1 - h) * ((self.GA + oA) * (1 - xc) + (self.GB + oB) * xc) + h * self.mu0
            mu = cb * (dG - cb * mt * q["dVm_alpha_dxB"])
        if sig:
            mu = mu - q["eps_iso_over_vB"] * (sig[0] + sig[1] + sig[2])
        Da, Dc = q["D_alpha"], q["D_compound"]
        x = torch.sigmoid(Y).clamp(1e-12, 1 - 1e-12)
        ld = x * (1 - x)
        mDY = float((((1 - h) * Da + h * Dc) * ld).mean())
        mk = self.mask * self.fwd(mu)
        dmu = 0.0
        xp, xm = (xc + 1e-5).clamp(1e-12, 1 - 1e-12), (xc - 1e-5).clamp(1e-12, 1 - 1e-12)
        (aP, bP), (aM, bM) = self.off(xp), self.off(xm)
        dmu = ((bP - bM) - (aP - aM)) / (xp - xm)

        def meff(D, g):
            return torch.minimum(D / g.clamp(min=1e-4), D * 1000.0)

        if gp:
            M = (1 - h) * (1 - _h(eta)) * meff(torch.full_like(h, Da), dmu / Vm)
        else:
            M = meff((1 - h) * Da + h * Dc, cb * dmu)
        div = 0.0
        for a in range(3):
            div = div + 1j * self.k[a] * self.fwd(M * self.inv(1j * self.k[a] * mk))
        if zm:
            src = _hp(pn) * ((pp - pn) / dt) * (vB - x) + ((1 - _h(pn)) * ld - 1) * dYdt
        else:
            src = ((_h(pp) - _h(pn)) / dt) * (vB - x) + ((1 - _h(pp)) * ld - 1) * dYdt
        Yn = self.inv(self.mask * (self.fwd(Y) + dt / (1 + dt * mDY * self.k2) * (div - self.fwd(src))))
        return Yn if zm else Yn.clamp(-20, 20)


def _read_params():
    prm = {}
    with open(PARAMS) as f:
        for line in f:
            line = line.split("#")[0].strip()
            if line:
                k, v = line.split("=")
                prm[k.strip()] = float(v)
    return prm


def _exact_dynamics(case, seed):
    if case["y_mode"] != "lagged":
        return None
    phi, xB, eta = _fields(case, seed)
    shape = tuple(phi.shape)
    gp, zm = case["model"] == "gp_zone", case["zero_mode"]
    prm = _read_params()
    m = _Model(shape, prm, hetero=case["elastic"] == "hetero")
    if not gp:
        eta = torch.zeros_like(phi)
    Y, dYdt = torch.logit(xB), torch.zeros_like(phi)
    vB = prm["v_B"]
    target = float(((1 - _h(phi)) * xB + vB * _h(phi)).sum())
    xof = torch.sigmoid if zm else (lambda y: torch.sigmoid(y.clamp(-20, 20)).clamp(1e-8, 1 - 1e-8))
    rows = []
    for _ in range(case["steps"]):
        x, el, sig = xof(Y), None, None
        if case["elastic"] != "off":
            e, e0, h = m.elastic(phi, x)
            el = [a - b for a, b in zip(e, e0)]
            sig = m.stress(el, h)
            del e, e0
        Ldt = prm["L_phi"] * m.dt
        pp = m.allen_cahn(phi - Ldt * m.phi_rhs(phi, x, el, sig), Ldt, prm["kappa_phi"]).clamp(-1e-6, 1 + 1e-6)
        en = eta
        if gp:
            Ldt = prm["gp_L_eta_code"] * m.dt
            en = m.allen_cahn(eta - Ldt * m.eta_rhs(eta, pp, x), Ldt, prm["gp_kappa_eta_code"]).clamp(0, 1)
        Yn = m.y_update(Y, dYdt, phi, pp, en, sig, gp, zm)
        if zm:
            a, lam = 1 - _h(pp), 0.0
            rest = float((_h(pp) * vB).sum())
            for _ in range(30):
                s = torch.sigmoid(Yn + lam)
                d = (float((a * s).sum()) + rest - target) / float((a * s * (1 - s)).sum())
                lam -= d
                if abs(d) < 1e-15 * max(1.0, abs(lam)):
                    break
            Yn = Yn + lam
        dYdt = (Yn - Y) / m.dt
        phi, eta, Y = pp, en, Yn
        if case["diag"]:
            x, h = xof(Y), _h(phi)
            rows.append([float(_h(phi.clamp(0, 1)).mean()), float(((1 - h) * x + h * vB).mean()), float(x.mean())])
    out = {"phi": phi, "xB": xof(Y)}
    if gp:
        out["eta"] = eta
    if case["diag"]:
        out["rows"] = torch.tensor(rows, dtype=F64)
    return out


def _exact_minimize(case, seed):
    phi, xB, e00 = _fields(case, seed)
    prm = _read_params()
    m = _Model(tuple(phi.shape), prm, eps00=e00, dt=0.05)
    V0, cap, lam_v = 0.1, 2.0, 0.0
    Ldt, kappa = prm["L_phi"] * m.dt, prm["kappa_phi"]
    Y, dYdt = torch.logit(xB), torch.zeros_like(phi)
    xof = (lambda y: torch.sigmoid(y.clamp(-20, 20)).clamp(1e-8, 1 - 1e-8))

    def gradient(p, x, el, sig):
        lap = m.inv(-(m.mask * m.k2) * m.fwd(p))
        ge = m.phi_rhs(p, x, el, sig)
        hp = _hp(p)
        return ge, lap, float(-(hp * (ge - kappa * lap)).sum() / (hp * hp).sum())

    def constrained(p, ge, lam):
        return m.allen_cahn(p - Ldt * (ge + lam * _hp(p)), Ldt, kappa).clamp(-1e-6, 1 + 1e-6)

    for _ in range(case["steps"]):
        x = xof(Y)
        e, e0, h = m.elastic(phi, x.clamp(max=cap))
        el = [a - b for a, b in zip(e, e0)]
        sig = m.stress(el, h)
        fs = 0.0
        for a in range(3):
            g = (torch.roll(phi, -1, a) - torch.roll(phi, 1, a)) * 0.5
            fs = fs + 0.5 * kappa * g * g
        F_surf = float((fs + prm["W"] * (phi * (1 - phi)) ** 2).mean())
        F_el = float(sum((0.5 if a < 3 else 1.0) * sig[a] * el[a] for a in range(6)).mean())

        def strain_at(p):     # the drive's elastic strain at phi, strain and stress frozen, composition uncapped
            return [a - b for a, b in zip(e, m.eigen(p, x))]

        ge, _, lraw = gradient(phi, x, strain_at(phi), sig)
        lam_v = 0.8 * lam_v + 0.2 * lraw
        pp = constrained(phi, ge, lam_v)
        sigY = m.stress([a - b for a, b in zip(e, m.eigen(phi, x.clamp(max=cap)))], h)
        Yn = m.y_update(Y, dYdt, phi, pp, None, sigY, False, False)
        dYdt = (Yn - Y) / m.dt
        Y, x = Yn, xof(Yn)
        ge, _, lam_v = gradient(pp, x, strain_at(pp), sig)
        pp = constrained(pp, ge, lam_v)
        mh, hp = float(_h(pp.clamp(0, 1)).mean()), _hp(pp)
        if abs(V0 - mh) > 1e-14:
            pp = (pp + (V0 - mh) / float((hp * hp).mean()) * hp).clamp(0, 1)
        phi = pp
        cap = 0.07 if float(x.max()) > 0.07 + 1e-12 else 2.0
    return {"phi": phi, "xB": xof(Y), "mean_h": float(_h(phi.clamp(0, 1)).mean()), "F_surf": F_surf, "F_el": F_el}


def _fno_exact(case, w, x):
    n, m = case["n"], case["modes"]
    ix = torch.tensor(list(range(m)) + list(range(n - m, n)), device="cuda")
    v = torch.einsum("oc,cxyz->oxyz", w["P"], x.double() * torch.tensor(FNO_IN, dtype=torch.float32, device="cuda")
                     .double()[:, None, None, None]) + w["p"][:, None, None, None]
    for i in range(case["layers"]):
        f = torch.fft.rfftn(v, dim=(1, 2, 3), norm="forward")[:, ix][:, :, ix][:, :, :, :m]
        R = torch.view_as_complex(w["R%d" % i].contiguous()).reshape(32, 32, 2 * m, 2 * m, m)
        g = torch.zeros((32, n, n, n // 2 + 1), dtype=C128, device="cuda")
        g[:, ix[:, None, None], ix[None, :, None], torch.arange(m, device="cuda")[None, None, :]] = \
            torch.einsum("ixyz,ioxyz->oxyz", f, R)
        v = torch.fft.irfftn(g, s=(n, n, n), dim=(1, 2, 3), norm="forward") \
            + torch.einsum("oc,cxyz->oxyz", w["W%d" % i], v) + w["b%d" % i][:, None, None, None]
        if i + 1 < case["layers"]:
            v = torch.nn.functional.gelu(v)
    v = torch.nn.functional.gelu(torch.einsum("oc,cxyz->oxyz", w["Q1"], v) + w["q1"][:, None, None, None])
    v = torch.einsum("oc,cxyz->oxyz", w["Q2"], v) + w["q2"][:, None, None, None]
    return v * torch.tensor(FNO_OUT, dtype=torch.float32, device="cuda").double()[:, None, None, None]


def _exact_fno(case, seed):
    # the model evaluates its weight blocks in bfloat16, its biases in float32
    w = {k: (v.bfloat16() if v.dim() > 1 else v).double() for k, v in _fno_weights(case, seed).items()}
    pairs = [_fno_pair(case, seed + 77 * i) for i in range(case.get("pairs", 1))]
    if case["kind"] == "fno":
        with torch.no_grad():
            return _fno_exact(case, w, pairs[0][0])
    for v in w.values():
        v.requires_grad_(True)
    losses = []
    for x, t in pairs:
        t = t.double()
        loss = ((_fno_exact(case, w, x) - t) ** 2).sum() / (t * t).sum()
        loss.backward()
        losses.append(float(loss))
    return {"grad": torch.cat([w[k].grad.reshape(-1) for k, _ in _fno_layout(case)]), "loss": losses}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fft":
        x = _real(case, seed)
        if case["op"] == "c2r":
            return torch.fft.irfftn(torch.fft.rfftn(x).to(C128), s=x.shape, norm="forward")
        return torch.fft.rfftn(x.double())
    if kind == "dynamics":
        with torch.no_grad():
            return _exact_dynamics(case, seed)
    if kind == "minimize":
        with torch.no_grad():
            return _exact_minimize(case, seed)
    if kind == "sweep":
        return None       # each of its cases is a minimize case; the sweep is held to the start's results
    return _exact_fno(case, seed)
