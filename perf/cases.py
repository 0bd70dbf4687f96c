"""The measured work of the wave path: what its users run, through the public
entry points of ``neuralmech_gb300``.

  forward     ``wave_forward``: modelling of a survey, 2D and 3D, FP32 or FP16 fields
  gradient    ``misfit_gradient``: one FWI iteration's misfit and gradient
  autograd    ``wave_forward`` under ``torch.autograd`` with a trace cotangent
  batch       ``BatchFWI``: gradients of several models of uneven size, one graph
  vd          ``vd_misfit_gradient``: the variable-density gradient
  steps       the single-step and eight-step kernels of the order-2 drivers
  imaging     ``analytic_signal`` and ``tfm`` on a captured full matrix

Models are layers with Gaussian anomalies and a small random perturbation of
every cell, seeded. Observed traces are direct arrivals of another speed with
a weak reflection, at the amplitude of modelled ones, so that the residual is
of the size of the data, as in the early iterations of an inversion.
``exact`` restates each path in plain FP64 torch: forward, exact adjoint by
transposition, no checkpoints.
"""
import math

import numpy as np
import torch

from neuralmech_gb300 import Grid
from neuralmech_gb300.batch import BatchFWI
from neuralmech_gb300.imaging import analytic_signal, tfm
from neuralmech_gb300.wavefd import (misfit_gradient, step2d_mixed_fast, step2d_order2, temporal_step_fast,
                                     vd_misfit_gradient, wave_forward)

DEV = "cuda"
DX = 10.0

_SURVEY = {"kind": "forward", "ndim": 2, "ny": 1, "nsrc": 1, "order": 8, "sponge": 20, "fields": "fp32", "hz": 22.0}
_FWI = {"kind": "gradient", "ndim": 2, "ny": 1, "nsrc": 1, "order": 8, "sponge": 20, "ckpt": "bf16", "step_block": 0,
        "kept": 0.0, "wavelet_gradient": False, "hz": 22.0}


def listed():
    return [
        # one shot on a small grid: what a first script, a test or a plate model runs; launches and latency
        dict(_SURVEY, name="forward_256_1shot", nz=256, nx=256, nshot=1, nt=1000, nrec=256),
        # one shot on a large grid: the throughput run of the forward solver
        dict(_SURVEY, name="forward_2048_1shot", nz=2048, nx=2048, nshot=1, nt=1000, nrec=2048),
        # a survey line modelled in one call, sides no multiple of any tile
        dict(_SURVEY, name="forward_401x1203_24shots", nz=401, nx=1203, nshot=24, nt=600, nrec=301),
        # an FWI iteration of a surface survey, two steps per launch, half of the levels kept in spare memory
        dict(_FWI, name="gradient_1024_32shots", nz=1024, nx=1024, nshot=32, nt=400, nrec=1024, step_block=2, kept=0.5),
        # the plate inversion: a small Dirichlet plate, few emitters, FP32 checkpoints
        dict(_FWI, name="gradient_plate_187x243_4shots", nz=187, nx=243, nshot=4, nt=500, nrec=32, sponge=0, ckpt="fp32"),
        # a differentiable forward inside a training loop: the default options, gradients of model and wavelet
        dict(_FWI, name="autograd_320x650_1shot", kind="autograd", nz=320, nx=650, nshot=1, nt=600, nrec=160, ckpt="fp32",
             wavelet_gradient=True),
        # several models of uneven size in one replayed graph, default checkpoints
        dict(_FWI, name="batch_4models", kind="batch", nmodel=4, nz=512, nx=1024, nshot=20, nt=240, nrec=512, step_block=2),
        # 3D modelling on odd sides, two shots
        dict(_SURVEY, name="forward3d_97x131x149_2shots", ndim=3, nz=97, ny=131, nx=149, nshot=2, nt=200, nrec=400,
             sponge=12),
        # 3D FWI iteration with BF16 checkpoints
        dict(_FWI, name="gradient3d_144x128x160_4shots", ndim=3, nz=144, ny=128, nx=160, nshot=4, nt=160, nrec=1024),
        # variable-density FWI iteration
        dict(_FWI, name="vd_gradient_480x760_12shots", kind="vd", nz=480, nx=760, nshot=12, nt=240, nrec=380, ckpt="fp32"),
        # the order-2 driver with eight steps per launch on its own grid
        {"name": "steps_temporal_8000x16000", "kind": "steps", "op": "temporal", "nz": 8000, "nx": 16000, "launches": 4},
        # full matrix capture to image: 32 elements, the plate driver's samples and pixels
        {"name": "imaging_32elements", "kind": "imaging", "elements": 32, "nt": 1500, "pixels": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; cell-steps bounded by the listed case of its kind."""
    what = rng.choice(["forward", "forward", "forward", "gradient", "gradient", "gradient", "autograd", "batch",
                       "forward3d", "gradient3d", "vd", "steps", "imaging"])
    order = rng.choice([8, 8, 8, 4, 2])
    if what == "forward":
        c = dict(_SURVEY, nz=_log(rng, 64, 2100), nx=_log(rng, 64, 2100), order=order, sponge=rng.choice([0, 12, 20]),
                 nrec=_log(rng, 1, 600), nsrc=rng.choice([1, 1, 3]), fields=rng.choice(["fp32", "fp32", "fp32", "fp16"]))
        c["nshot"] = max(1, min(_log(rng, 1, 48), int(12e6 // (c["nz"] * c["nx"]))))
        c["nt"] = max(100, min(_log(rng, 200, 1200), int(4e9 // (c["nz"] * c["nx"] * c["nshot"]))))
        return c
    if what in ("gradient", "autograd"):
        c = dict(_FWI, kind=what, nz=_log(rng, 100, 1100), nx=_log(rng, 100, 1100), order=order, sponge=rng.choice([0, 12, 20]),
                 nrec=_log(rng, 8, 600), ckpt=rng.choice(["bf16", "fp32", "i16"]), step_block=rng.choice([0, 2]),
                 kept=rng.choice([0.0, 0.0, 0.5, 1.0]), wavelet_gradient=rng.choice([False, True]))
        c["nshot"] = max(1, min(_log(rng, 1, 40), int(30e6 // (c["nz"] * c["nx"]))))
        c["nt"] = max(80, min(_log(rng, 150, 700), int(6e9 // (c["nz"] * c["nx"] * c["nshot"]))))
        return c
    if what == "batch":
        return dict(_FWI, kind="batch", nmodel=rng.randint(2, 5), nz=_log(rng, 200, 500), nx=_log(rng, 600, 1000),
                    nshot=rng.randint(6, 20), nt=rng.randint(100, 240), nrec=_log(rng, 32, 500), order=order,
                    step_block=rng.choice([0, 2]))
    if what in ("forward3d", "gradient3d"):
        base = _SURVEY if what == "forward3d" else _FWI
        c = dict(base, ndim=3, nz=_log(rng, 48, 160), ny=_log(rng, 48, 160), nx=_log(rng, 48, 200), order=order,
                 sponge=rng.choice([0, 12, 20]), nrec=_log(rng, 16, 1024))
        c["nshot"] = max(1, min(rng.randint(1, 4), int(10e6 // (c["nz"] * c["ny"] * c["nx"]))))
        c["nt"] = max(100, min(rng.randint(100, 200), int(1.2e9 // (c["nz"] * c["ny"] * c["nx"] * c["nshot"]))))
        return c
    if what == "vd":
        c = dict(_FWI, kind="vd", nz=_log(rng, 80, 700), nx=_log(rng, 80, 900), order=order, ckpt=rng.choice(["fp32", "bf16"]),
                 nrec=_log(rng, 8, 380), wavelet_gradient=rng.choice([False, True]))
        c["nshot"] = max(1, min(rng.randint(1, 14), int(4.3e6 // (c["nz"] * c["nx"]))))
        c["nt"] = max(60, min(rng.randint(120, 400), int(1e9 // (c["nz"] * c["nx"] * c["nshot"]))))
        return c
    if what == "steps":
        return {"kind": "steps", "op": rng.choice(["temporal", "order2", "mixed"]), "nz": _log(rng, 200, 8000),
                "nx": _log(rng, 200, 15000), "launches": rng.randint(1, 4)}
    return {"kind": "imaging", "elements": rng.randint(8, 32), "nt": rng.randint(400, 1500), "pixels": _log(rng, 64, 512)}


# ---------------------------------------------------------------- inputs
def _shape(c):
    return (c["nz"], c["nx"]) if c.get("ndim", 2) == 2 else (c["nz"], c["ny"], c["nx"])


def _model(shape, seed, top=1500.0, bottom=3200.0):
    """Layers with depth, three Gaussian anomalies of +/- 8 %, 0.5 % noise."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    axes = torch.meshgrid(*[torch.linspace(0, 1, n, device=DEV) for n in shape], indexing="ij")
    v = top + (bottom - top) * torch.floor(axes[0] * 4) / 4
    for k in range(3):
        p = torch.rand(len(shape) + 1, generator=g, device=DEV)
        r2 = sum((a - 0.1 - 0.8 * q) ** 2 for a, q in zip(axes, p))
        v = v * (1 + (0.08 if k % 2 else -0.08) * torch.exp(-r2 / (2 * (0.04 + 0.1 * p[-1]) ** 2)))
    return (v * (1 + 0.005 * torch.randn(shape, generator=g, device=DEV))).float().contiguous()


def _ricker(hz, nt, dt):
    a = (math.pi * hz * (np.arange(nt) * dt - 1.5 / hz)) ** 2
    return (1 - 2 * a) * np.exp(-a)


def _line(n, lo, hi):
    return np.rint(np.linspace(lo, hi, n)).astype(np.int32)


def _acquisition(c, R):
    """Sources and receivers near the top surface, (nshot, n, ndim)."""
    shape, S = _shape(c), c["nshot"]
    lo, zs = R + 1, min(R + 2, shape[0] - R - 1)
    n1 = shape[-1] - R - 2
    if len(shape) == 2:
        xs = _line(S, lo, n1) if S > 1 else np.array([shape[1] // 2], np.int32)
        src = np.stack([np.stack([np.full(S, zs, np.int32), np.clip(xs + 7 * k, lo, n1)], -1) for k in range(c["nsrc"])], 1)
        rec = np.stack([np.full(c["nrec"], zs, np.int32), _line(c["nrec"], lo, n1)], -1)
    else:
        xs = _line(S, shape[2] // 4, 3 * shape[2] // 4)
        ys = _line(S, 3 * shape[1] // 4, shape[1] // 4)
        src = np.stack([np.full(S, zs, np.int32), ys, xs], -1)[:, None, :]
        k = max(1, int(math.isqrt(c["nrec"])))
        ry, rx = np.meshgrid(_line(k, lo, shape[1] - R - 2), _line(k, lo, n1), indexing="ij")
        rec = np.stack([np.full(k * k, zs, np.int32), ry.ravel(), rx.ravel()], -1)
    return src.astype(np.int32), np.broadcast_to(rec, (S,) + rec.shape).astype(np.int32).copy()


def _survey(c, seed):
    """(velocity, wavelet (S, nt, nsrc), src, rec, grid) of a case."""
    shape = _shape(c)
    vel = _model(shape, seed)
    # a step that FP32 holds exactly, inside the order-8 bounds for every seed of the generator
    dt = float(np.float32((0.44 if len(shape) == 2 else 0.36) * DX / 4000.0))
    g = np.random.default_rng(seed)
    w = np.stack([_ricker(c["hz"] * f, c["nt"], dt) for f in g.uniform(0.9, 1.1, c["nshot"])])
    w = w[:, :, None] * g.uniform(0.7, 1.3, (c["nshot"], 1, c["nsrc"]))
    src, rec = _acquisition(c, c["order"] // 2)
    kw = {}
    if c["kind"] != "forward":
        kw = {"ckpt_format": c["ckpt"], "step_block": c["step_block"], "store_levels": int(c["kept"] * c["nt"])}
    elif len(shape) == 2:
        kw = {"field_format": c["fields"]}
    grid = Grid(shape, (DX,) * len(shape), dt, c["nt"], order=c["order"], sponge=c["sponge"], **kw)
    return vel, torch.from_numpy(w.astype(np.float32)).to(DEV), src, rec, grid


def _observed(c, grid, src, rec, wav, seed):
    """Arrivals of another model: a direct wave and a weak later one per trace, (S, nt, nrec)."""
    v = 1450.0 + 100.0 * np.random.default_rng(seed + 1).random()
    t = torch.arange(grid.nt, device=DEV, dtype=torch.float32)[None, :, None] * grid.dt
    r = torch.from_numpy(np.sqrt(((rec - src[:, :1]).astype(np.float64) ** 2).sum(-1))).float().to(DEV)[:, None, :] * DX
    amp = (18.0 if len(grid.shape) == 2 else 3.0) / (r / DX + 8.0) ** (0.5 if len(grid.shape) == 2 else 1.0)
    out = torch.zeros((src.shape[0], grid.nt, rec.shape[1]), device=DEV)
    for tau, a in ((r / v, 1.0), (torch.sqrt(r * r + (0.6 * grid.shape[0] * DX) ** 2) / v + 0.05, 0.2)):
        x = (math.pi * c["hz"] * (t - tau - 1.5 / c["hz"])) ** 2
        out += a * amp * (1 - 2 * x) * torch.exp(-x)
    return out.contiguous()


def _parts(c, seed):
    """The models of a batch: sides, steps and shots vary about the case's."""
    rng = np.random.default_rng(c["nz"] * 7 + c["nx"])
    parts = []
    for k in range(c["nmodel"]):
        n = dict(c, kind="gradient")
        n["nz"], n["nx"] = (int(s * f) for s, f in zip((c["nz"], c["nx"]), rng.uniform(0.6, 1.0, 2)))
        n["nt"] = int(c["nt"] * rng.uniform(0.7, 1.0))
        n["nshot"] = c["nshot"] // c["nmodel"] + (k < c["nshot"] % c["nmodel"])
        parts.append((n, seed + 1000 * k))
    return parts


def _pulses(c, seed):
    """Two levels of the order-2 drivers' field: Gaussian pulses at rest, rows padded to 32."""
    N, M = c["nz"], c["nx"]
    Mp = (M + 32) // 32 * 32
    p = torch.rand((4, 2), generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)
    x, y = torch.linspace(0, 1, N, device=DEV)[:, None], torch.linspace(0, 2, M, device=DEV)[None, :]
    u = torch.zeros((N, Mp), device=DEV)
    for a, b in p.tolist():
        u[:, :M] += torch.exp(-(x - 0.2 - 0.6 * a) ** 2 / (2 * 0.02 ** 2)) * torch.exp(-(y - 0.4 - 1.2 * b) ** 2 / (2 * 0.03 ** 2))
    u[0], u[N - 1], u[:, 0], u[:, M - 1:] = 0, 0, 0, 0
    dx, dy = 1.0 / (N - 1), 2.0 / (M - 1)
    return u, (1.0, 0.9 * min(dx, dy) / math.sqrt(2), dx, dy, N, M)


def _matrix(c, seed):
    """Full-matrix traces of point scatterers, (E, nt, E), with the array and the image grid."""
    E, nt, dt, v = c["elements"], c["nt"], 2.5 / (c["nt"] - 1), 1.0
    xs = np.linspace(0.1, 0.9, E)
    el = np.stack([xs, np.full(E, 0.01)], -1)
    g = np.random.default_rng(seed)
    t = torch.arange(nt, device=DEV, dtype=torch.float64)[None, :, None] * dt
    h = 1e-3 * torch.randn((E, nt, E), generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV, dtype=torch.float64)
    for px, py in g.uniform(0.2, 0.8, (4, 2)):
        d = torch.from_numpy(np.hypot(el[:, 0] - px, el[:, 1] - py)).to(DEV)
        tau = t - (d[:, None, None] + d[None, None, :]) / v - 0.05
        h += torch.sin(2 * math.pi * 20.0 * tau) * torch.exp(-(tau / 0.03) ** 2)
    px = torch.linspace(0, 1, c["pixels"], device=DEV)
    X, Y = torch.meshgrid(px, px, indexing="ij")
    return h.float().contiguous(), el.astype(np.float32), dt, v, X.contiguous(), Y.contiguous()


def _vd_media(vel):
    """(kappa, rho): density following the speed, smooth contrasts."""
    rho = 1000.0 + 0.35 * (vel - 1400.0)
    return (rho * vel * vel).contiguous(), rho.contiguous()


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "steps":
        u, args = _pulses(c, seed)
        u = u.half() if c["op"] == "mixed" else u
        return {"case": c, "u": u, "bufs": [torch.zeros_like(u) for _ in range(4)], "args": args}
    if kind == "imaging":
        h, el, dt, v, X, Y = _matrix(c, seed)
        return {"case": c, "h": h, "el": el, "dt": dt, "v": v, "X": X, "Y": Y}
    if kind == "batch":
        models = []
        for n, s in _parts(c, seed):
            vel, wav, src, rec, grid = _survey(n, s)
            models.append(dict(vel=vel, wavelet=wav, src=src, rec=rec, observed=_observed(n, grid, src, rec, wav, s), grid=grid))
        return {"case": c, "batch": BatchFWI(models, autotune=False)}
    vel, wav, src, rec, grid = _survey(c, seed)
    s = {"case": c, "vel": vel, "wav": wav, "src": src, "rec": rec, "grid": grid}
    if kind != "forward":
        s["obs"] = _observed(c, grid, src, rec, wav, seed)
    if kind == "vd":
        s["kappa"], s["rho"] = _vd_media(vel)
    if kind == "autograd":
        s["vel"] = vel.requires_grad_(True)
        s["wav"] = wav.requires_grad_(c["wavelet_gradient"])
    return s


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "forward":
        return wave_forward(s["vel"], s["wav"], s["src"], s["rec"], s["grid"])
    if kind == "gradient":
        return misfit_gradient(s["vel"], s["wav"], s["src"], s["rec"], s["obs"], s["grid"],
                               want_wavelet=c["wavelet_gradient"], want_traces=True)
    if kind == "autograd":
        traces = wave_forward(s["vel"], s["wav"], s["src"], s["rec"], s["grid"])
        of = [s["vel"]] + ([s["wav"]] if c["wavelet_gradient"] else [])
        return [traces.detach(), *torch.autograd.grad(traces, of, traces.detach() - s["obs"])]
    if kind == "batch":
        misfits, grads = s["batch"].run()
        return [misfits, *grads]
    if kind == "vd":
        return vd_misfit_gradient(s["kappa"], s["rho"], s["wav"], s["src"], s["rec"], s["obs"], s["grid"],
                                  want_wavelet=c["wavelet_gradient"])
    if kind == "steps":
        a, b, (p, q, r, t) = s["u"], s["u"], s["bufs"]
        for _ in range(c["launches"]):
            if c["op"] == "temporal":
                temporal_step_fast(a, b, p, q, *s["args"])
                a, b, p, q, r, t = p, q, r, t, p, q
            else:
                (step2d_order2 if c["op"] == "order2" else step2d_mixed_fast)(a, b, p, *s["args"])
                a, b, p, q, r, t = b, p, q, r, t, p
        return [a, b]
    return tfm(analytic_signal(s["h"].permute(0, 2, 1).contiguous()), s["el"], 0.05, s["dt"], s["v"], s["X"], s["Y"])


def work(case):
    """Inputs read and outputs written once; FLOPs of the stencil updates (a fused multiply-add is 2)."""
    c, kind = case, case["kind"]
    if kind == "steps":
        cells, steps = c["nz"] * c["nx"], c["launches"] * (8 if c["op"] == "temporal" else 1)
        return {"bytes": cells * (2 if c["op"] == "mixed" else 4) * 4.0, "flops": cells * steps * 10.0}
    if kind == "imaging":
        E, nt, px = c["elements"], c["nt"], c["pixels"] ** 2
        return {"bytes": 4.0 * (E * E * nt + 3 * px), "flops": E * E * 5.0 * nt * math.log2(nt) * 2 + px * E * (E + 1) / 2 * 16.0}
    if kind == "batch":
        each = [work(n) for n, _ in _parts(c, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    cells, R, nd = math.prod(_shape(c)), c["order"] // 2, len(_shape(c))
    lap = 3.0 * R * nd + 1
    if kind == "vd":  # two staggered differences per axis
        lap = 2 * nd * 3.0 * R + nd
    updates = cells * c["nshot"] * c["nt"]
    traces = 4.0 * c["nshot"] * c["nt"] * c["nrec"]
    if kind == "forward":
        return {"bytes": 4.0 * cells + traces, "flops": updates * (lap + 4)}
    return {"bytes": (4.0 if kind == "vd" else 2.0) * 4 * cells + 2 * traces, "flops": updates * (2 * (lap + 4) + lap + 2)}


# ---------------------------------------------------------------- the same in FP64
def _second(order):
    R = order // 2
    f = math.factorial
    a = [0.0] + [2.0 * (1 if k % 2 else -1) * f(R) ** 2 / (k * k * f(R - k) * f(R + k)) for k in range(1, R + 1)]
    a[0] = -2.0 * sum(a)
    return a


def _staggered(R):
    c = []
    for k in range(1, R + 1):
        v = 1.0 / (2 * k - 1)
        for m in range(1, R + 1):
            if m != k:
                v *= (2 * m - 1) ** 2 / ((2 * m - 1) ** 2 - (2 * k - 1) ** 2)
        c.append(v)
    return c


def _damping(grid, dev):
    """g on the whole grid: the product of the axes' exponential tapers (as FP32 profiles)."""
    g = torch.ones(grid.shape, dtype=torch.float64, device=dev)
    W = grid.sponge
    for ax, n in enumerate(grid.shape):
        p = np.ones(n)
        for d in range(1, W + 1):
            for i in (W - d, n - 1 - (W - d)):
                if 0 <= i < n:
                    p[i] = math.exp(-((grid.sponge_strength / W) * d) ** 2)
        view = [1] * len(grid.shape)
        view[ax] = n
        g = g * torch.from_numpy(p.astype(np.float32).astype(np.float64)).to(dev).view(view)
    return g


class _Plain:
    """The recursion of one medium in FP64: u_{n+1} = g (2 u + k A u + s w) - g^2 u_{n-1} on the interior."""

    def __init__(self, grid, vel, src, rec, rho=None):
        self.dev, self.grid, self.R, nd = vel.device, grid, grid.order // 2, len(grid.shape)
        R, dt = self.R, float(np.float32(grid.dt))
        self.inner = tuple(slice(R, n - R) for n in grid.shape)
        self.full = tuple(grid.shape)
        self.g = _damping(grid, self.dev)
        self.vel, self.rho = vel.double(), None if rho is None else rho.double()
        self.k = (self.vel * dt / DX) ** 2 if rho is None else self.vel * dt * dt / (DX * DX)
        self.a, self.c = _second(grid.order), _staggered(R)
        if rho is not None:
            b = 1.0 / self.rho
            self.bh = [0.5 * (b.narrow(ax, 0, b.shape[ax] - 1) + b.narrow(ax, 1, b.shape[ax] - 1)) for ax in range(nd)]
        self.src = [torch.from_numpy(src[..., d].astype(np.int64)).to(self.dev) for d in range(nd)]
        self.rec = [torch.from_numpy(rec[..., d].astype(np.int64)).to(self.dev) for d in range(nd)]

    def at(self, pos, shots):
        s = torch.arange(shots.start, shots.stop, device=self.dev)[:, None]
        return (s - shots.start,) + tuple(p[shots] for p in pos)

    def half(self, u, ax):
        """D u at the half points j + 1/2, j = 0 .. n - 2, of an axis (u zero outside)."""
        R, n, ax1 = self.R, u.shape[ax + 1], ax + 1
        pad = [0, 0] * (len(self.full) - 1 - ax) + [R, R]
        p = torch.nn.functional.pad(u, pad)
        out = torch.zeros_like(u.narrow(ax1, 0, n - 1))
        for k, c in enumerate(self.c, 1):
            out.add_(p.narrow(ax1, R + k, n - 1) - p.narrow(ax1, R - k + 1, n - 1), alpha=c)
        return out

    def apply(self, u):
        """A u on the interior."""
        R, off = self.R, 1
        I = (slice(None),) + self.inner
        if self.rho is None:
            out = u[I] * (self.a[0] * len(self.full))
            for ax, n in enumerate(self.full):
                for k in range(1, R + 1):
                    for s in (-k, k):
                        J = list(I)
                        J[ax + off] = slice(R + s, n - R + s)
                        out.add_(u[tuple(J)], alpha=self.a[k])
            return out
        out = torch.zeros_like(u[I])
        for ax, n in enumerate(self.full):
            f = self.half(u, ax) * self.bh[ax]
            J = list(I)
            J[ax + off] = slice(None)
            f = f[tuple(J)]
            for k, c in enumerate(self.c, 1):  # F_{i + k - 1/2} - F_{i - k + 1/2}
                out.add_(f.narrow(ax + off, R + k - 1, n - 2 * R) - f.narrow(ax + off, R - k, n - 2 * R), alpha=c)
        return out

    def forward(self, wav, shots, keep):
        """Traces of a range of shots, and every level when `keep`."""
        S, w = shots.stop - shots.start, wav[shots].double()
        I = (slice(None),) + self.inner
        g, k = self.g[self.inner], self.k[self.inner]
        up, u = (torch.zeros((S,) + self.full, dtype=torch.float64, device=self.dev) for _ in range(2))
        src, rec = self.at(self.src, shots), self.at(self.rec, shots)
        gs = self.g[src[1:]]
        levels, traces = [], []
        for n in range(self.grid.nt):
            if keep:
                levels.append(u)
            v = torch.zeros_like(u)
            v[I] = g * (2 * u[I] + k * self.apply(u)) - g * g * up[I]
            v.index_put_(src, gs * w[:, n], accumulate=True)
            up, u = u, v
            traces.append(u[rec])
        return torch.stack(traces, 1), levels

    def adjoint(self, levels, d, shots, sums):
        """Adds a range of shots' gradient to the sums; their wavelet gradients."""
        I = (slice(None),) + self.inner
        g, k = self.g[self.inner], self.k[self.inner]
        src, rec = self.at(self.src, shots), self.at(self.rec, shots)
        S = shots.stop - shots.start
        p1, p2 = (torch.zeros((S,) + self.full, dtype=torch.float64, device=self.dev) for _ in range(2))
        dw = [None] * self.grid.nt
        for n in range(self.grid.nt, 0, -1):  # the cotangent of u_n from those of u_{n+1}, u_{n+2}
            y = torch.zeros_like(p1)
            y[I] = g * p1[I]
            q = torch.zeros_like(p1)
            q[I] = 2 * y[I] - g * g * p2[I]
            y[I] *= k
            q[I] += self.apply(y)
            q.index_put_(rec, d[:, n - 1], accumulate=True)
            dw[n - 1] = self.g[src[1:]] * q[src]
            p2, p1 = p1, q
            # u_n = g (2 u + k A u) ... of u = u_{n-1}
            u = levels[n - 1]
            y = torch.zeros_like(q)
            y[I] = g * q[I]
            sums["k"][self.inner] += (y[I] * self.apply(u)).sum(0)
            if self.rho is not None:
                y[I] *= k
                for ax in range(len(self.full)):
                    sums[ax] -= (self.half(y, ax) * self.half(u, ax)).sum(0)
        return torch.stack(dw, 1)


def _exact_survey(c, vel, wav, src, rec, grid, obs=None, rho=None):
    p = _Plain(grid, vel, src, rec, rho)
    S, keep = wav.shape[0], obs is not None
    per = math.prod(grid.shape) * 8.0
    group = max(1, min(S, int(2.4e10 // (per * (grid.nt if keep else 8)))))
    sums = {"k": torch.zeros(grid.shape, dtype=torch.float64, device=vel.device)}
    if rho is not None:
        sums.update({ax: torch.zeros_like(b) for ax, b in enumerate(p.bh)})
    traces, dws = [], []
    for a in range(0, S, group):
        shots = slice(a, min(S, a + group))
        t, levels = p.forward(wav, shots, keep)
        traces.append(t)
        if keep:
            dws.append(p.adjoint(levels, t - obs[shots].double(), shots, sums))
    traces = torch.cat(traces)
    if not keep:
        return traces
    misfit = 0.5 * (traces - obs.double()).square().sum()
    dw = torch.cat(dws)
    if rho is None:
        return misfit, [sums["k"] * 2 * p.k / p.vel], dw, traces
    dt = float(np.float32(grid.dt))
    db = torch.zeros_like(p.rho)
    for ax in range(2):
        n = db.shape[ax]
        db.narrow(ax, 0, n - 1).add_(0.5 * sums[ax])
        db.narrow(ax, 1, n - 1).add_(0.5 * sums[ax])
    return misfit, [sums["k"] * dt * dt / (DX * DX), -db / p.rho ** 2], dw, traces


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "steps":
        if c["op"] == "mixed":
            return None  # every step rounds the field to FP16
        u, (v, dt, dx, dy, N, M) = _pulses(c, seed)
        dt, dx, dy = (float(np.float32(x)) for x in (dt, dx, dy))
        a, b = u.double(), u.double()
        ax, ay = v * v * dt * dt / (dx * dx), v * v * dt * dt / (dy * dy)
        older = None
        for _ in range(c["launches"] * (8 if c["op"] == "temporal" else 1)):
            n = torch.zeros_like(b)
            i = b[1:N - 1, 1:M - 1]
            n[1:N - 1, 1:M - 1] = (2 * i - a[1:N - 1, 1:M - 1] + ax * (b[:N - 2, 1:M - 1] - 2 * i + b[2:N, 1:M - 1])
                                   + ay * (b[1:N - 1, :M - 2] - 2 * i + b[1:N - 1, 2:M]))
            older, a, b = a, b, n
        return [a, b]
    if kind == "imaging":
        h, el, dt, v, X, Y = _matrix(c, seed)
        nt, E = c["nt"], c["elements"]
        x = h.permute(0, 2, 1).double()
        F = torch.fft.fft(x, dim=-1)
        m = torch.zeros(nt, dtype=torch.float64, device=DEV)
        m[0] = 1
        m[1:(nt + 1) // 2] = 2
        if nt % 2 == 0:
            m[nt // 2] = 1
        z = torch.fft.ifft(F * m, dim=-1)
        el64 = torch.from_numpy(el).double().to(DEV)
        px, py = X.reshape(-1).double(), Y.reshape(-1).double()
        out = torch.zeros(px.numel(), dtype=torch.complex128, device=DEV)
        far = [torch.hypot(px - e[0], py - e[1]) for e in el64]
        for e in range(E):
            for r in range(e, E):
                f = (0.05 + (far[e] + far[r]) / v) / dt
                i = torch.floor(f).long()
                ok = i < nt - 1
                i = i.clamp(0, nt - 2)
                w = f - i
                out += (1 if r == e else 2) * ok * (z[e, r][i] * (1 - w) + z[e, r][i + 1] * w)
        return out.abs().reshape(X.shape)
    if kind == "batch":
        got = []
        for n, s in _parts(c, seed):
            vel, wav, src, rec, grid = _survey(n, s)
            got.append(_exact_survey(n, vel, wav, src, rec, grid, _observed(n, grid, src, rec, wav, s)))
        return [torch.stack([g[0] for g in got]), *[g[1][0] for g in got]]
    vel, wav, src, rec, grid = _survey(c, seed)
    if kind == "forward":
        return _exact_survey(c, vel, wav, src, rec, grid)
    obs = _observed(c, grid, src, rec, wav, seed)
    kappa, rho = _vd_media(vel) if kind == "vd" else (vel, None)
    misfit, grads, dw, traces = _exact_survey(c, kappa, wav, src, rec, grid, obs, rho)
    more = [dw] if c["wavelet_gradient"] else []
    if kind == "autograd":
        return [traces, *grads, *more]
    return [misfit, *grads, *more] + ([traces] if kind == "gradient" else [])
