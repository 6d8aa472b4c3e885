"""Timed cases of the framework: one pass each through its public entry points.

  step      one RK3 step of dense device arrays (Dycore.advance), flat grid
  terrain   the same over a static terrain-following grid, Deardorff closure
  moving    the same over the travelling-wave grid, with acoustic substeps
  learned   the same with the tensor-core subgrid closure
  kessler   the standalone microphysics call on a view of the state
  train     minibatch Adam steps of the closure network
  infer     the closure network over a batch of cells

A state advances in place from pass to pass, as a host model's does.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os

import numpy as np
import torch

import erf_b200
from erf_b200 import cases as flows
from erf_b200 import config as C
from erf_b200 import terrain as hills
from erf_b200.closure import MLP, coarse_case, load_closure
from erf_b200.dycore import Dycore, dense_fab, load_library

NET_FILE = os.path.join(os.path.dirname(erf_b200.__file__), "data", "closure_abl.npz")
SCHEMES = {"u5": C.UPWIND_5TH, "u3": C.UPWIND_3RD, "w5": C.WENO_5, "w3": C.WENO_3}
TRAIN_LR = 2e-3
DEV = "cuda" if torch.cuda.is_available() else "cpu"   # (inputs and exact() need no GPU)


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _step(flow, nx, ny, nz, form="fp64", dyc="u5", dry="u5", moist="w5"):
    return {"kind": "step", "flow": flow, "nx": nx, "ny": ny, "nz": nz, "form": form, "dyc": dyc, "dry": dry,
            "moist": moist}


def listed():
    return [
        # a column-physics or unit-test sized box: launches and latency
        dict(_step("abl", 24, 20, 32), name="abl 24x20x32"),
        # the dry boundary layer of the tests and the benchmark
        dict(_step("abl", 64, 64, 64), name="abl 64x64x64"),
        # the headline moist bubble (Kessler, WENO5 scalars), in both forms
        dict(_step("bubble", 128, 128, 80, dry="w5"), name="bubble 128x128x80"),
        dict(_step("bubble", 128, 128, 80, form="mixed", dry="w5"), name="bubble 128x128x80 mixed"),
        # the reference's default schemes (Upwind_3rd, WENO3) on a box that no tile divides
        dict(_step("bubble", 157, 93, 61, dyc="u3", dry="u3", moist="w3"), name="bubble 157x93x61 defaults"),
        # the fine boundary layer that the closure's training data come from
        dict(_step("abl", 512, 512, 128), name="abl 512x512x128"),
        # the terrain boundary layer of the benchmark
        {"name": "terrain 256x256x96", "kind": "terrain", "nx": 256, "ny": 256, "nz": 96, "form": "fp64"},
        # the reference's moving-terrain test, 20 substeps a step
        {"name": "moving 40x8x79", "kind": "moving", "nx": 40, "ny": 8, "nz": 79},
        # the coarse boundary layer that the learned closure was trained for
        {"name": "learned 128x128x32", "kind": "learned", "nx": 128, "ny": 128, "nz": 32, "form": "mixed"},
        # microphysics called alone, as a host model with its own dynamics does
        {"name": "kessler 128x128x80", "kind": "kessler", "nx": 128, "ny": 128, "nz": 80, "rain": True},
        # the training loop's minibatch; inference over one coarse snapshot
        {"name": "train 8192x20", "kind": "train", "rows": 65536, "batch": 8192, "iters": 20},
        {"name": "infer 524288", "kind": "infer", "rows": 524288},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["terrain", "moving", "learned", "kessler", "train", "infer"])
    if kind == "step":
        flow = rng.choice(["abl", "bubble"])
        nx, ny, nz = _log(rng, 16, 400), _log(rng, 16, 400), _log(rng, 16, 128)
        return _step(flow, nx, ny, nz, form=rng.choice(["fp64", "fp64", "mixed"]), dyc=rng.choice(["u5", "u5", "u3"]),
                     dry=rng.choice(["u5", "w5", "u3"]), moist=rng.choice(["w5", "w5", "w3"]))
    if kind == "terrain":
        return {"kind": kind, "nx": _log(rng, 24, 256), "ny": _log(rng, 24, 256), "nz": _log(rng, 20, 96),
                "form": rng.choice(["fp64", "mixed"])}
    if kind == "moving":
        return {"kind": kind, "nx": _log(rng, 24, 200), "ny": _log(rng, 6, 64), "nz": _log(rng, 24, 96)}
    if kind == "learned":
        return {"kind": kind, "nx": _log(rng, 16, 160), "ny": _log(rng, 16, 160), "nz": _log(rng, 16, 48),
                "form": rng.choice(["fp64", "mixed"])}
    if kind == "kessler":
        return {"kind": kind, "nx": _log(rng, 16, 256), "ny": _log(rng, 16, 256), "nz": _log(rng, 16, 100),
                "rain": rng.choice([True, True, False])}
    if kind == "train":
        batch = _log(rng, 512, 16384)
        return {"kind": kind, "rows": batch * rng.randint(1, 8) + rng.randint(0, 100), "batch": batch,
                "iters": rng.randint(5, 40)}
    return {"kind": "infer", "rows": _log(rng, 2000, 2000000)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _noise(g, *shape):
    return 2.0 * torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64) - 1.0


def _flow(case):
    """The package's configuration and sounding of a flat case."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["kind"] == "learned":
        fl = coarse_case(flows.abl_fine(nx=4 * nx, ny=4 * ny, nz=4 * nz), 4)
        fl.cfg.les_type = C.LES_MLP
    elif case.get("flow") == "abl":
        fl = flows.abl_dry(nx=nx, ny=ny, nz=nz)
    else:
        fl = flows.moist_bubble(nx=nx, ny=ny, nz=nz)
        fl.cfg.dz = 20000.0 / nz
        fl.cfg.dt = min(2.0, 2.0 * fl.cfg.dz / 250.0)
        # the 20 km sounding of the benchmark's 80 levels at this case's levels
        deep = flows.moist_bubble(nx=4, ny=4, nz=80)
        z0, z = (np.arange(80) + 0.5) * 250.0, (np.arange(nz) + 0.5) * fl.cfg.dz
        fl.theta_cc, fl.qv_cc, fl.u_cc = (np.interp(z, z0, a) for a in (deep.theta_cc, deep.qv_cc, deep.u_cc))
    c = fl.cfg
    if case["kind"] == "step":
        c.dycore_horiz_adv = c.dycore_vert_adv = SCHEMES[case["dyc"]]
        c.dryscal_horiz_adv = c.dryscal_vert_adv = SCHEMES[case["dry"]]
        if c.moisture != C.MOIST_NONE:
            c.moistscal_horiz_adv = c.moistscal_vert_adv = SCHEMES[case["moist"]]
    if case["kind"] == "kessler" and not case["rain"]:
        c.moisture, c.ncomp, c.buoyancy_type = C.MOIST_KESSLER_NORAIN, 7, 1
    c.precision = C.PREC_MIXED if case.get("form") == "mixed" else C.PREC_FP64
    return fl


def _base(fl):
    """Hydrostatic base state of a sounding: rho0, p0, pi0, theta0 at k = -1 .. nz."""
    c, nz, g = fl.cfg, fl.cfg.nz, fl.cfg.gravity
    kap = C.R_D / C.CP_D

    def rho_of(th, p, q):
        return 1e5 ** kap * p ** (1 / 1.4) / (C.R_D * th * (1 + 461.505 / C.R_D * q))
    r0 = np.zeros(nz + 2)
    p, rho, zp, q = fl.p_sfc, rho_of(fl.theta_sfc, fl.p_sfc, fl.qv_sfc), 0.0, fl.qv_sfc
    for k in range(nz):
        z, th, qk = (k + 0.5) * c.dz, fl.theta_cc[k], fl.qv_cc[k]
        pk = p
        for _ in range(60):
            pk = p - 0.5 * g * (z - zp) * (rho * (1 + q) + rho_of(th, pk, qk) * (1 + qk))
        p, rho, zp, q = pk, rho_of(th, pk, qk), z, qk
        r0[k + 1] = rho
    r0[0], r0[-1] = r0[1], r0[-2]
    p0 = np.zeros(nz + 2)
    p0[0], p0[1] = 1e5 + 0.5 * c.dz * r0[1] * g, 1e5 - 0.5 * c.dz * r0[1] * g
    for k in range(2, nz + 2):
        p0[k] = p0[k - 1] - c.dz * 0.5 * (r0[k] + r0[k - 1]) * g
    pi0 = (p0 / 1e5) ** (C.R_D / c.c_p)
    th0 = (p0 * 1e5 ** 0.4) ** (1 / 1.4) / C.R_D / r0
    return [r0, p0, pi0, th0]


def _fields(case, fl, base, seed):
    """A seeded flow: the sounding with a bubble or a noisy boundary layer, and turbulence in all three winds."""
    c, g = fl.cfg, _gen(seed)
    nx, ny, nz = c.nx, c.ny, c.nz

    def col(a):
        return torch.as_tensor(np.asarray(a), device=DEV, dtype=torch.float64)[:, None, None]
    z = (np.arange(nz) + 0.5) * c.dz
    low = col(np.where(z < 0.25 * nz * c.dz, 1.0, 0.1))
    theta = col(fl.theta_cc) + 0.1 * low * _noise(g, nz, ny, nx)
    cons = torch.zeros(c.ncomp, nz, ny, nx, device=DEV, dtype=torch.float64)
    rho = col(base[0][1:nz + 1])
    if c.moisture != C.MOIST_NONE:
        x = (torch.arange(nx, device=DEV) + 0.5) / nx - 0.5
        y = (torch.arange(ny, device=DEV) + 0.5) / ny - 0.5
        r2 = (4 * x[None, None, :]) ** 2 + (4 * y[None, :, None]) ** 2 + col(((z - 1500.0) / 1500.0) ** 2)
        warm = torch.exp(-2 * r2)
        theta = theta + 3.0 * warm
        cons[5] = rho * col(fl.qv_cc) * (1.0 + 0.1 * warm + 0.02 * _noise(g, nz, ny, nx))
        cons[6] = rho * 1e-3 * warm * (1.0 + 0.5 * _noise(g, nz, ny, nx))
        if c.ncomp > 7:
            cons[7] = rho * 5e-4 * warm * (1.0 + 0.5 * _noise(g, nz, ny, nx))
    cons[0] = rho
    cons[1] = rho * theta
    cons[4] = rho * (1.0 + 0.1 * _noise(g, nz, ny, nx))
    # (the learned closure's coarse noise is the fine run's, block averaged)
    amp = 0.06 if case["kind"] == "learned" else 0.5
    u = torch.empty(nz, ny, nx + 1, device=DEV, dtype=torch.float64)
    v = torch.empty(nz, ny + 1, nx, device=DEV, dtype=torch.float64)
    w = torch.zeros(nz + 1, ny, nx, device=DEV, dtype=torch.float64)
    u[:, :, :nx] = col(fl.u_cc) + amp * low * _noise(g, nz, ny, nx)
    v[:, :ny] = 0.3 * col(fl.u_cc) + amp * low * _noise(g, nz, ny, nx)
    u[:, :, nx], v[:, ny] = u[:, :, 0], v[:, 0]
    w[1:nz] = amp * low[1:] * _noise(g, nz - 1, ny, nx)
    return cons, u, v, w


@functools.lru_cache(maxsize=2)
def _hill(nx, ny, nz):
    """Grid and base state of a terrain case (they do not depend on the seed)."""
    # the benchmark's hill (300 m high, 800 m wide on 6.4 km), lower where the box is smaller or shallower
    top = 5.0 * (1.04 ** nz - 1.0) / 0.04
    r0 = 0.125 * 25.0 * min(nx, ny)
    h0 = min(300.0, 0.2 * top, 0.375 * r0)
    t = hills.abl_terrain(nx=nx, ny=ny, nz=nz, dt=0.25, h0=h0, r0=r0, amp=h0 / 15.0)
    dy = Dycore(t.cfg)
    dy.set_terrain(t.z_nd)
    base = dy.make_base_state_terrain(t)
    dy.close()
    return t, base, [torch.from_numpy(a) for a in t.build_state(base[0])]


@functools.lru_cache(maxsize=2)
def _wave(nx, ny, nz):
    """The travelling wave is uniform in y: four rows of it, repeated."""
    t = hills.moving_terrain(nx=nx, ny=4, nz=nz, Lx=5.0 * nx, Ly=20.0, H=400.0 * nz / 79, substeps=True)
    base = [np.repeat(b.reshape(nz + 2, 4, nx)[:, :1], ny, axis=1).reshape(-1) for b in t.base]
    cons, u, v, w = t.build_state()
    state = [np.repeat(cons[:, :, :1], ny, axis=2), np.repeat(u[:, :1], ny, axis=1),
             np.repeat(v[:, :1], ny + 1, axis=1), np.repeat(w[:, :1], ny, axis=1)]
    cfg = t.cfg.copy()
    cfg.ny, cfg.dy = ny, 5.0
    return cfg, base, [torch.from_numpy(np.ascontiguousarray(a)) for a in state]


def _net_inputs(case, seed):
    g = _gen(seed)
    x = torch.randn(case["rows"], 13, generator=g, device=DEV)
    a = torch.randn(13, 9, generator=g, device=DEV) / 4.0
    t = torch.tanh(x @ a) + 0.1 * x[:, :9] ** 2
    t = ((t - t.mean(0)) / t.std(0)).contiguous()
    n = [64 * 16, 64 * 64, 64 * 64, 16 * 64]
    scale = [(2 / 13) ** 0.5, (2 / 64) ** 0.5, (2 / 64) ** 0.5, (1 / 64) ** 0.5]
    w = [torch.randn(m, generator=g, device=DEV) * s for m, s in zip(n, scale)]
    w[0].view(64, 16)[:, 13:] = 0
    w[3].view(16, 64)[9:] = 0
    b = [0.1 * torch.randn(64, generator=g, device=DEV) for _ in range(3)]
    b.append(torch.zeros(16, device=DEV))
    return x, t, torch.cat(w + b)


def _net_scaling():
    """Per-feature and per-output scaling of the inference cases."""
    q = np.arange(13)
    return 0.1 * (q - 6.0), 0.5 + 0.1 * q, 0.01 * np.arange(9.0), 0.2 + 0.05 * np.arange(9.0)


@functools.lru_cache(maxsize=None)
def _stream():
    """The program's compute stream: every state's work is ordered on it."""
    return torch.cuda.Stream()


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("train", "infer"):
        x, t, p = _net_inputs(case, seed)
        net = MLP()
        net.set_params(p.cpu().numpy())
        net.set_normalization(*(_net_scaling() if kind == "infer" else
                                (np.zeros(13), np.ones(13), np.zeros(9), np.ones(9))))
        s.update(net=net, x=x, t=t, case=case, y=torch.zeros(case["rows"], 9, device=DEV))
        torch.cuda.synchronize()
        return s
    handle = _stream().cuda_stream
    if kind == "terrain":
        t, base, state = _hill(case["nx"], case["ny"], case["nz"])
        cfg = t.cfg.copy()
        cfg.precision = C.PREC_MIXED if case["form"] == "mixed" else C.PREC_FP64
        dy = Dycore(cfg, handle)
        dy.set_terrain(t.z_nd)
    elif kind == "moving":
        cfg, base, state = _wave(case["nx"], case["ny"], case["nz"])
        dy = Dycore(cfg, handle)
    else:
        fl = _flow(case)
        base = _base(fl)
        dy = Dycore(fl.cfg, handle)
        state = _fields(case, fl, base, seed)
    dy.set_base_state(base)
    if kind in ("terrain", "moving"):
        cons, u, v, w = (a.cuda() for a in state)
        g = _gen(seed)
        cons[1] *= 1.0 + 1e-4 * _noise(g, *cons[1].shape)
        cons[4] = cons[0] * (1.0 + 0.1 * _noise(g, *cons[0].shape))
        if kind == "terrain":
            u[:, :, :-1] += 0.5 * _noise(g, *u[:, :, :-1].shape)
            v[:, :-1] += 3.0 + 0.5 * _noise(g, *v[:, :-1].shape)
            u[:, :, -1], v[:, -1] = u[:, :, 0], v[:, 0]
            w[1:-1] += 0.5 * _noise(g, *w[1:-1].shape)
        state = cons, u, v, w
    if kind == "learned":
        s["net"] = load_closure(NET_FILE, handle)
        dy.set_closure(s["net"])
    s.update(dy=dy, state=state)
    if kind == "kessler":
        cfg = dy.cfg
        s["fab"] = dense_fab(state[0], 0, cfg.nx, cfg.ny, cfg.nz, cfg.ncomp)
        s["dt"] = cfg.dt
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "train":
        c = s["case"]
        loss = s["net"].train(s["x"], s["t"], c["rows"], c["batch"], c["iters"], TRAIN_LR)
        return {"loss": loss, "params": s["net"].get_params()}
    if kind == "infer":
        s["net"].infer(s["x"], s["y"], s["case"]["rows"])
        return s["y"]
    if kind == "kessler":
        if load_library().erf_b200_kessler_advance(s["dy"].ctx, ctypes.byref(s["fab"]), s["dt"]):
            raise RuntimeError("erf_b200_kessler_advance failed")
        return [q for q in s["state"][0]]
    s["dy"].advance(*s["state"], 1)
    cons, u, v, w = s["state"]
    return {"cons": [cons[n] for n in range(cons.shape[0])], "u": u, "v": v, "w": w}


# ---------------------------------------------------------------------------
# Work and tolerances
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    net_flops = 2 * (13 * 64 + 2 * 64 * 64 + 64 * 9)
    if kind == "infer":
        n = case["rows"]
        return {"bytes": n * 4 * (13 + 9), "flops": n * net_flops}
    if kind == "train":
        n = case["batch"] * case["iters"]
        return {"bytes": n * 4 * (13 + 9) + case["iters"] * 10448 * 4 * 6, "flops": 3 * n * net_flops}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "kessler":
        # rho, rho theta and the species in, all but rho out
        nq = 3 if case["rain"] else 2
        return {"bytes": cells * 8 * (2 + nq + 1 + nq), "flops": cells * 300}
    # a step reads its state once and writes it once; the operations are those of three slow right-hand sides
    # (face interpolants of three momenta and the scalars), ten substeps and the closure
    moist = kind == "step" and case["flow"] == "bubble"
    ncomp = 8 if moist else 5
    slow = 3 * 3 * (25 if not moist else 60) * (5 + (3 if moist else 0))
    sub = 41 if kind == "moving" else 10
    closure = 3 * net_flops if kind == "learned" else (0 if moist or kind == "moving" else 150)
    return {"bytes": cells * 8 * 2 * (ncomp + 3), "flops": cells * (slow + sub * 60 + closure)}


def tolerance(case):
    """About four times the largest error seen against exact() over drawn cases, by kind."""
    kind = case["kind"]
    if kind == "train":
        return {"rel": 4e-3, "max": 0.1}       # BF16 products under Adam's sign-like first steps
    if kind == "infer":
        return {"rel": 2.5e-2, "max": 0.25}    # BF16 products
    if kind == "kessler":
        return {"rel": 1e-12, "max": 4e-11}
    if kind == "learned":
        return {"rel": 8e-4, "max": 1e-2}      # BF16 stresses; w moves by this share in a step
    if case.get("form") == "mixed":
        return {"rel": 1.2e-5, "max": 1e-4}    # FP32 tendencies and increments of an FP64 state
    if kind == "step":
        return {"rel": 4e-12, "max": 4e-11}    # w over two steps; the other fields are 1e-14
    # (no exact() here: the bars that the framework's own tests hold these grids to)
    return {"rel": 1e-10, "max": 1e-8}


# ---------------------------------------------------------------------------
# The same in plain torch, FP64: one step on a flat grid, Kessler, the network.
# (The terrain grids have none: their metric terms alone would restate most of
# the framework's own oracle.)
# ---------------------------------------------------------------------------
def _x(a, n):
    return torch.roll(a, -n, -1)


def _y(a, n):
    return torch.roll(a, -n, -2)


def _pad(a, n, zero_lo=False, zero_hi=False):
    """n ghost levels at either end: the end level again, or 0."""
    lo, hi = a[:1].repeat(n, 1, 1), a[-1:].repeat(n, 1, 1)
    return torch.cat([lo * 0 if zero_lo else lo, a, hi * 0 if zero_hi else hi])


def _weno(v, scheme):
    eps = 1e-6
    if scheme == C.WENO_3:
        a, b, c = v[1:4]
        g = [(1 / 3, (b - a) ** 2, (3 * b - a) / 2), (2 / 3, (c - b) ** 2, (b + c) / 2)]
    else:
        a, b, c, d, e = v
        g = [(0.1, 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2, (2 * a - 7 * b + 11 * c) / 6),
             (0.6, 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2, (-b + 5 * c + 2 * d) / 6),
             (0.3, 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2, (2 * c + 5 * d - e) / 6)]
    wt = [q / (eps + b) ** 2 for q, b, _ in g]
    return sum(w * p for w, (_, _, p) in zip(wt, g)) / sum(wt)


def _face(scheme, s, a):
    """Value on a face from the six cells around it (s[2] below, s[3] above), carried by a."""
    if scheme in (C.WENO_3, C.WENO_5):
        up = a > 1e-12
        v = [torch.where(up, s[m], s[5 - m]) for m in range(5)]
        return torch.where(a.abs() > 1e-12, _weno(v, scheme), 0.5 * (s[2] + s[3]))
    sg = torch.sign(a)
    if scheme == C.UPWIND_3RD:
        return (7 * (s[3] + s[2]) - (s[4] + s[1]) + sg * ((s[4] - s[1]) - 3 * (s[3] - s[2]))) / 12
    return (37 * (s[3] + s[2]) - 8 * (s[4] + s[1]) + (s[5] + s[0])
            - sg * ((s[5] - s[0]) - 5 * (s[4] - s[1]) + 10 * (s[3] - s[2]))) / 60


def _along(shift, f):
    return [shift(f, m) for m in range(-3, 3)]


def _up(p, n):
    return [p[m:m + n] for m in range(6)]


class _Flat:
    def __init__(self, cfg, base):
        self.c = cfg
        self.dxi, self.dyi, self.dzi = 1 / cfg.dx, 1 / cfg.dy, 1 / cfg.dz
        self.r0, self.p0, self.pi0 = (torch.as_tensor(b, device=DEV)[:, None, None] for b in base[:3])
        self.moist = cfg.moisture != C.MOIST_NONE
        self.lo0, self.hi0 = cfg.zlo_bc == C.BC_NO_SLIP_WALL, cfg.zhi_bc == C.BC_NO_SLIP_WALL
        self.kap = C.R_D / cfg.c_p

    def pres(self, rt, qv=0.0):
        return 1e5 * (C.R_D * rt * (1 + 461.505 / C.R_D * qv) / 1e5) ** 1.4

    def div(self, fx, fy, fz):
        return (_x(fx, 1) - fx) * self.dxi + (_y(fy, 1) - fy) * self.dyi + (fz[1:] - fz[:-1]) * self.dzi

    def scalar(self, phi, mx, my, mz, scheme):
        nz = phi.shape[0]
        return -self.div(mx * _face(scheme, _along(_x, phi), mx), my * _face(scheme, _along(_y, phi), my),
                         mz * _face(scheme, _up(_pad(phi, 3), nz + 1), mz))

    def strain(self, u, v, w):
        dxi, dyi, dzi = self.dxi, self.dyi, self.dzi
        s11, s22, s33 = (_x(u, 1) - u) * dxi, (_y(v, 1) - v) * dyi, (w[1:] - w[:-1]) * dzi
        s12 = 0.5 * ((u - _y(u, -1)) * dyi + (v - _x(v, -1)) * dxi)

        def vert(t, ws):
            p = _pad(t, 1, self.lo0, self.hi0)
            d = (p[1:] - p[:-1]) * dzi
            if self.lo0:
                d[0] = (3 * t[0] - t[1] / 3) * dzi
            if self.hi0:
                d[-1] = -(3 * t[-1] - t[-2] / 3) * dzi
            return 0.5 * (d + ws)
        return s11, s22, s33, s12, vert(u, (w - _x(w, -1)) * dxi), vert(v, (w - _y(w, -1)) * dyi)

    def viscosity(self, rho, u, v, w):
        s11, s22, s33, s12, s13, s23 = self.strain(u, v, w)
        e12 = 0.25 * (s12 + _y(s12, 1) + _x(s12, 1) + _x(_y(s12, 1), 1))
        e13 = 0.25 * (s13[:-1] + s13[1:] + _x(s13[:-1] + s13[1:], 1))
        e23 = 0.25 * (s23[:-1] + s23[1:] + _y(s23[:-1] + s23[1:], 1))
        ss = s11 ** 2 + s22 ** 2 + s33 ** 2 + 2 * (e12 ** 2 + e13 ** 2 + e23 ** 2)
        c = self.c
        return c.Cs ** 2 * (c.dx * c.dy * c.dz) ** (2 / 3) * rho * torch.sqrt(2 * ss)

    def stress(self, mu, u, v, w):
        s11, s22, s33, s12, s13, s23 = self.strain(u, v, w)
        er = (s11 + s22 + s33) / 3
        p = _pad(mu, 1)
        m12 = 0.25 * (mu + _x(mu, -1) + _y(mu, -1) + _x(_y(mu, -1), -1))
        m13, m23 = (0.25 * (q[1:] + q[:-1]) for q in (p + _x(p, -1), p + _y(p, -1)))
        return [-2 * mu * (s11 - er), -2 * mu * (s22 - er), -2 * mu * (s33 - er), -2 * m12 * s12, -2 * m13 * s13,
                -2 * m23 * s23]

    def diffuse(self, mu, phi, inv):
        p, m = _pad(phi, 1), _pad(mu, 1)
        return self.div(-0.5 * inv * (mu + _x(mu, -1)) * (phi - _x(phi, -1)) * self.dxi,
                        -0.5 * inv * (mu + _y(mu, -1)) * (phi - _y(phi, -1)) * self.dyi,
                        -0.5 * inv * (m[1:] + m[:-1]) * (p[1:] - p[:-1]) * self.dzi)

    def network(self, rho, theta, u, v, w, net):
        """Cell stresses and heat fluxes of the learned closure, Smagorinsky outside its training range."""
        c = self.c
        hx, hy = 0.5 * self.dxi, 0.5 * self.dyi
        uc, vc, wc = 0.5 * (u + _x(u, 1)), 0.5 * (v + _y(v, 1)), 0.5 * (w[1:] + w[:-1])

        def dz(a):
            p = _pad(a, 1)
            d = (p[2:] - p[:-2]) * 0.5 * self.dzi
            d[0], d[-1] = 2 * d[0], 2 * d[-1]
            return d

        def dx(a):
            return (_x(a, 1) - _x(a, -1)) * hx

        def dy(a):
            return (_y(a, 1) - _y(a, -1)) * hy
        delta = (c.dx * c.dy * c.dz) ** (1 / 3)
        f = torch.stack([(_x(u, 1) - u) * self.dxi, dy(uc), dz(uc), dx(vc), (_y(v, 1) - v) * self.dyi, dz(vc), dx(wc),
                         dy(wc), (w[1:] - w[:-1]) * self.dzi, dx(theta), dy(theta), dz(theta),
                         torch.full_like(rho, delta)], -1)
        d = {k: torch.as_tensor(net[k].astype(np.float64), device=DEV) for k in
             ("params", "in_mean", "in_std", "out_mean", "out_std", "in_lo", "in_hi")}
        m = 0.05 * (d["in_hi"] - d["in_lo"])
        edge = torch.minimum(f.float().double() - d["in_lo"], d["in_hi"] - f.float().double())
        wgt = torch.where(m > 0, (edge / torch.where(m > 0, m, torch.ones_like(m))).clamp(0, 1),
                          (edge >= 0).double()).amin(-1, keepdim=True)
        y = _forward(d["params"], (f - d["in_mean"]) / d["in_std"]) * d["out_std"] + d["out_mean"]
        s12, s13, s23 = 0.5 * (f[..., 1] + f[..., 3]), 0.5 * (f[..., 2] + f[..., 6]), 0.5 * (f[..., 5] + f[..., 7])
        s11, s22, s33 = f[..., 0], f[..., 4], f[..., 8]
        ss = s11 ** 2 + s22 ** 2 + s33 ** 2 + 2 * (s12 ** 2 + s13 ** 2 + s23 ** 2)
        nut, tr = (c.Cs * delta) ** 2 * torch.sqrt(2 * ss), (s11 + s22 + s33) / 3
        sm = torch.stack([-2 * nut * (s11 - tr), -2 * nut * (s22 - tr), -2 * nut * (s33 - tr), -2 * nut * s12,
                          -2 * nut * s13, -2 * nut * s23] + [-nut / c.Pr_t * f[..., q] for q in (9, 10, 11)], -1)
        y = rho[..., None] * (wgt * y + (1 - wgt) * sm)
        t11, t22, t33, c12, c13, c23, qx, qy, qz = y.unbind(-1)
        p13, p23, pz = _pad(c13, 1), _pad(c23, 1), _pad(qz, 1)
        t12 = 0.25 * (c12 + _x(c12, -1) + _y(c12, -1) + _x(_y(c12, -1), -1))
        t13 = 0.25 * (p13[1:] + p13[:-1] + _x(p13[1:] + p13[:-1], -1))
        t23 = 0.25 * (p23[1:] + p23[:-1] + _y(p23[1:] + p23[:-1], -1))
        fz = 0.5 * (pz[1:] + pz[:-1])
        fz[0] = fz[-1] = 0
        return [t11, t22, t33, t12, t13, t23], self.div(0.5 * (qx + _x(qx, -1)), 0.5 * (qy + _y(qy, -1)), fz)

    def momentum(self, cons, prim, pp, u, v, w, mx, my, mz, tau):
        c, nz = self.c, u.shape[0]
        dxi, dyi, dzi, sch = self.dxi, self.dyi, self.dzi, self.c.dycore_horiz_adv
        rho = cons[0]

        def lo(a, sh):
            return 0.5 * (a + sh(a, -1))

        def tangential(f, sh):
            a, b, d = lo(mx, sh), lo(my, sh), lo(mz, sh)
            return -self.div(a * _face(sch, _along(_x, f), a), b * _face(sch, _along(_y, f), b),
                             d * _face(sch, _up(_pad(f, 3, self.lo0, self.hi0), nz + 1), d))
        # (div takes the high face one cell up in x and y)
        fu, fv = tangential(u, _x), tangential(v, _y)
        az = 0.5 * (mz[1:] + mz[:-1])                # between faces k and k + 1
        wp = _pad(w, 2)
        s = [wp[m:m + nz] for m in range(6)]          # faces k - 2 .. k + 3 about the middle of cell k
        fz = _face(sch, s, az)
        c4 = (7 * (s[2] + s[3]) - (s[1] + s[4])) / 12
        for k in (1, nz - 2):
            if sch != C.UPWIND_3RD:
                fz[k] = c4[k]
        for k in (0, nz - 1):
            fz[k] = 0.5 * (w[k] + w[k + 1])
        fz = az * fz
        ax, ay = 0.5 * (mx[1:] + mx[:-1]), 0.5 * (my[1:] + my[:-1])
        wi = w[1:-1]
        hx, hy = ax * _face(sch, _along(_x, wi), ax), ay * _face(sch, _along(_y, wi), ay)
        fw = -((_x(hx, 1) - hx) * dxi + (_y(hy, 1) - hy) * dyi + (fz[1:] - fz[:-1]) * dzi)
        if tau:
            t11, t22, t33, t12, t13, t23 = tau
            fu = fu - ((t11 - _x(t11, -1)) * dxi + (_y(t12, 1) - t12) * dyi + (t13[1:] - t13[:-1]) * dzi)
            fv = fv - ((_x(t12, 1) - t12) * dxi + (t22 - _y(t22, -1)) * dyi + (t23[1:] - t23[:-1]) * dzi)
            a, b = t13[1:-1], t23[1:-1]
            fw = fw - ((_x(a, 1) - a) * dxi + (_y(b, 1) - b) * dyi + (t33[1:] - t33[:-1]) * dzi)
        q = prim[4] + prim[5] if self.moist else torch.zeros_like(rho)
        su, sv = lo(rho, _x) * c.abl_geo_forcing[0], lo(rho, _y) * c.abl_geo_forcing[1]
        r0, g = self.r0[1:-1], c.gravity
        if not self.moist:
            b = -g * 0.5 * ((rho - r0)[1:] + (rho - r0)[:-1])
        elif c.buoyancy_type == 1:
            b = rho + sum(cons[5:]) - r0
            b = -g * 0.5 * (b[1:] + b[:-1])
        else:
            m = [a.mean((1, 2), keepdim=True) for a in [rho, prim[0]] + list(prim[4:7])]
            tm = self.pres(m[0] * m[1], m[2]) / (C.R_D * m[0] * (1 + 461.505 / C.R_D * m[2]))
            t = self.pres(cons[1], prim[4]) / (C.R_D * rho * (1 + 461.505 / C.R_D * prim[4]))
            e = (0.61 * (prim[4] - m[2]) - (prim[5] - m[3] + prim[6] - m[4])
                 + (t - tm) / tm * (1 + 0.61 * m[2] - m[3] - m[4]))
            b = g * 0.25 * (e[1:] + e[:-1]) * (m[0][1:] + m[0][:-1])
        sw = b + 0.5 * (rho[1:] + rho[:-1]) * c.abl_geo_forcing[2]
        if c.use_coriolis:
            vb = 0.5 * (my + _y(my, 1))
            wb = 0.5 * (mz[1:] + mz[:-1])
            ub = 0.5 * (mx + _x(mx, 1))
            su = su + c.coriolis_factor * (lo(vb, _x) * c.sinphi - lo(wb, _y) * c.cosphi)
            sv = sv - c.coriolis_factor * lo(ub, _y) * c.sinphi
            sw = sw + c.coriolis_factor * 0.5 * (ub[1:] + ub[:-1]) * c.cosphi
        fu = fu - (pp - _x(pp, -1)) * dxi / (1 + lo(q, _x)) + su
        fv = fv - (pp - _y(pp, -1)) * dyi / (1 + lo(q, _y)) + sv
        fw = fw + (sw - (pp[1:] - pp[:-1]) * dzi) / (1 + 0.5 * (q[1:] + q[:-1]))
        z = torch.zeros_like(fw[:1])
        return fu, fv, torch.cat([z, fw, z])

    def step(self, cons, u, v, w, net=None):
        c, nz = self.c, u.shape[0]
        dxi, dyi, dzi, hg = self.dxi, self.dyi, self.dzi, 0.5 * c.gravity
        b1, b2 = 0.45, 0.55
        w = w.clone()
        w[0] = w[-1] = 0

        def lo(a, sh):
            return 0.5 * (a + sh(a, -1))

        def facez(a):
            p = _pad(a, 1)
            return 0.5 * (p[1:] + p[:-1])
        old = [cons, u * lo(cons[0], _x), v * lo(cons[0], _y), w * facez(cons[0])]
        mu = self.viscosity(cons[0], u, v, w) if c.les_type != C.LES_NONE else None
        stage = old
        for nrk, (nsub, dtau, dt) in enumerate([(1, c.dt / 3, c.dt / 3), (c.mri_ratio // 2, c.dt / c.mri_ratio, c.dt / 2),
                                                (c.mri_ratio, c.dt / c.mri_ratio, c.dt)]):
            S, sx, sy, sz = stage
            prim = [S[n] / S[0] for n in range(1, c.ncomp)]
            th = prim[0]
            qv = prim[4] if self.moist else 0.0
            pi = (C.R_D * S[1] / 1e5) ** (1.4 * self.kap)
            pp = self.pres(S[1], qv) - self.p0[1:-1]
            fr = -self.div(sx, sy, sz)
            ft = self.scalar(th, sx, sy, sz, c.dycore_horiz_adv)
            tau = None
            if net is not None:
                tau, heat = self.network(S[0], th, u, v, w, net)
                ft = ft - heat
            elif mu is not None:
                tau = self.stress(mu, u, v, w)
                ft = ft - self.diffuse(mu, th, 1 / c.Pr_t)
            fu, fv, fw = self.momentum(S, prim, pp, u, v, w, sx, sy, sz, tau)
            # implicit coefficients on the interior faces
            i, r0, pi0 = slice(1, nz), self.r0, self.pi0
            q = prim[4] + prim[5] if self.moist else torch.zeros_like(th)
            wet = 1 + 0.5 * (q[1:] + q[:-1])
            pic, cv = 0.5 * (pi[1:] + pi[:-1]), c.c_p - C.R_D
            cP = (-1.4 * C.R_D * dzi + hg * C.R_D * r0[2:nz + 1] / (cv * pi0[2:nz + 1] * S[1][1:])) * pic / wet
            cQ = (1.4 * C.R_D * dzi + hg * C.R_D * r0[1:nz] / (cv * pi0[1:nz] * S[1][:-1])) * pic / wet
            thf = facez(th)
            D = dtau * dtau * b2 * b2 * dzi
            A, Cc = D * (hg - cQ * thf[:-2]), D * (-hg + cP * thf[2:])
            B = 1 + D * (cQ - cP) * thf[1:-1]
            av = [sx.clone(), sy.clone(), sz.clone()]
            new, lag = [old[0][0], old[0][1]] + old[1:], None
            for ks in range(nsub):
                drt = new[1] - S[1]
                ex = drt if lag is None else drt + 0.1 * (drt - lag)
                lag = drt
                gx, gy = (ex - _x(ex, -1)) * dxi, (ex - _y(ex, -1)) * dyi
                if nrk == 0:
                    gx, gy = 0 * gx, 0 * gy
                dx_ = new[2] - sx + dtau * (fu - 1.4 * C.R_D * lo(pi, _x) * gx / (1 + lo(q, _x)))
                dy_ = new[3] - sy + dtau * (fv - 1.4 * C.R_D * lo(pi, _y) * gy / (1 + lo(q, _y)))
                t0 = (_x(dx_, 1) - dx_) * dxi + (_y(dy_, 1) - dy_) * dyi
                tx, ty = dx_ * lo(th, _x), dy_ * lo(th, _y)
                t1 = (_x(tx, 1) - tx) * dxi + (_y(ty, 1) - ty) * dyi
                om = new[4] - sz
                dr = new[0] - S[0]
                r = cP * drt[1:] + cQ * drt[:-1] - hg * (dr[1:] + dr[:-1])
                r1 = hg * (-fr[1:] - fr[:-1] + t0[1:] + t0[:-1]) + cP * (ft[1:] - t1[1:]) + cQ * (ft[:-1] - t1[:-1])
                ot = om * thf
                r1 = r1 + b1 * dzi * ((om[2:] - om[:-2]) * hg - (ot[2:] - ot[1:-1]) * cP - (ot[1:-1] - ot[:-2]) * cQ)
                rhs = om[i] + dtau * (fw[i] + r + dtau * b2 * r1)
                # Thomas; 0 on the walls
                sol, gam = torch.zeros_like(om), torch.zeros_like(om)
                for k in range(1, nz):
                    bet = B[k - 1] - A[k - 1] * gam[k - 1]
                    gam[k] = Cc[k - 1] / bet
                    sol[k] = (rhs[k - 1] - A[k - 1] * sol[k - 1]) / bet
                for k in range(nz - 1, 0, -1):
                    sol[k] -= gam[k] * sol[k + 1]
                z = b2 * sol + b1 * om
                for a, d in zip(av, (dx_, dy_, z)):
                    a += d / nsub
                zt = z * thf
                new = [new[0] + dtau * (fr - t0 - dzi * (z[1:] - z[:-1])),
                       new[1] + dtau * (ft - t1 - dzi * (zt[1:] - zt[:-1])), sx + dx_, sy + dy_, sz + sol]
            out = S.clone()
            out[0], out[1] = new[0], new[1]
            for n in [4] + list(range(5, c.ncomp)):
                f = self.scalar(prim[n - 1], *av, c.dryscal_horiz_adv if n == 4 else c.moistscal_horiz_adv)
                if mu is not None:
                    f = f - self.diffuse(mu, prim[n - 1], 1 / c.Sc_t)
                out[n] = cons[n] + dt * f
                if n > 4:
                    out[n].clamp_(min=0)
            stage = [out] + new[2:]
            u, v, w = new[2] / lo(out[0], _x), new[3] / lo(out[0], _y), new[4] / facez(out[0])
        out = stage[0]
        return (_kessler(c, out) if self.moist else out), u, v, w


def _kessler(c, cons):
    rho, rt = cons[0], cons[1]
    qv, qc = cons[5] / rho, cons[6] / rho
    rain = c.moisture == C.MOIST_KESSLER
    qp = cons[7] / rho if rain else torch.zeros_like(rho)
    th, rv = rt / rho, 461.505 / C.R_D
    p = 1e5 * (C.R_D * rt * (1 + rv * qv) / 1e5) ** 1.4
    t, mb = p / (C.R_D * rho * (1 + rv * qv)), p / 100

    def fall(ra, qa):
        qa = qa.clamp(min=0)
        f = ra * 36.34 * (ra * 0.001 * qa) ** 0.1346 * (ra / 1.16) ** -0.5 * qa
        return torch.where(f.abs() < 1e-14, 0.0, f)

    def mid(a):
        return torch.cat([a[:1], 0.5 * (a[1:] + a[:-1]), a[-1:]])
    fz = fall(mid(rho), mid(qp)) if rain else torch.zeros_like(mid(rho))
    d, e = (t - 273.16).clamp(max=70.0), t - 273.16
    es, ds = torch.zeros_like(t), torch.zeros_like(t)
    # Flatau et al. (1992), saturation over water
    for k in (-0.976195544e-15, -0.952447341e-13, 0.640689451e-10, 0.206739458e-7, 0.302950461e-5, 0.264847430e-3,
              0.142986287e-1, 0.443987641, 6.11239921):
        es = es * d + k
    for k in (-0.599634321e-17, -0.792933209e-14, -0.604119582e-12, 0.385208005e-9, 0.103167413e-6, 0.121167162e-4,
              0.794747212e-3, 0.285976452e-1, 0.443956472):
        ds = ds * e + k
    ds = torch.where(e >= 70, 0.0, ds)
    rr = C.R_D / 461.505
    qs = rr * es / torch.maximum(es, mb - es)
    fac = 2.0 + 2.5e6 / C.CP_D * rr * ds / mb
    if rain:
        qv, qp, qs = qv.clamp(min=0), qp.clamp(min=0), qs.clamp(min=0)
    qc = qc.clamp(min=0)
    cond = torch.where(qv > qs, torch.minimum(qv, (qv - qs) / fac), 0.0)
    evap = torch.where((qv < qs) & (qc > 0), torch.minimum(qc, (qs - qv) / fac), 0.0)
    zero = torch.zeros_like(rho)
    r2v = c2r = zero
    if rain:
        rq = 0.001 * rho * qp
        r2v = (1 - qv / qs) * (1.6 + 124.9 * rq ** 0.2046) * rq ** 0.525 / (5.4e5 + 2.55e6 / (mb * qs)) * c.dt / (0.001 * rho)
        r2v = torch.where((qp > 0) & (qv < qs), torch.minimum(qp, r2v), zero)
        c2r = c.dt * (2.2 * qp ** 0.875 * qc + torch.where(qc > 1e-3, 1e-3 * (qc - 1e-3), zero))
        c2r = torch.where(qc > 0, torch.minimum(c2r, qc), zero)
    sed = c.dt / rho * (fz[1:] - fz[:-1]) / c.dz
    sed = torch.where(sed.abs() < 1e-14, zero, sed)
    th = th + th / t * 2.501e6 / c.c_p * (cond - evap - r2v)
    out = cons.clone()
    out[1] = rho * th
    out[5] = rho * (qv - cond + evap + r2v).clamp(min=0)
    out[6] = rho * (qc + cond - evap - c2r).clamp(min=0)
    if rain:
        out[7] = rho * (qp + sed + c2r - r2v).clamp(min=0)
    return out


def _forward(p, x):
    o = [0, 1024, 5120, 9216, 10240, 10304, 10368, 10432, 10448]
    w = [p[o[0]:o[1]].view(64, 16)[:, :13], p[o[1]:o[2]].view(64, 64), p[o[2]:o[3]].view(64, 64),
         p[o[3]:o[4]].view(16, 64)[:9]]
    b = [p[o[4]:o[5]], p[o[5]:o[6]], p[o[6]:o[7]], p[o[7]:o[8]][:9]]
    for q in range(3):
        x = torch.nn.functional.gelu(x @ w[q].T + b[q], approximate="tanh")
    return x @ w[3].T + b[3]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("terrain", "moving"):
        return None
    if kind == "infer":
        x, _, p = _net_inputs(case, seed)
        im, istd, om, ostd = (torch.as_tensor(a, device=DEV) for a in _net_scaling())
        return _forward(p.double(), (x.double() - im) / istd) * ostd + om
    if kind == "train":
        x, t, p = _net_inputs(case, seed)
        p = p.double().requires_grad_()
        opt = torch.optim.Adam([p], lr=TRAIN_LR, betas=(0.9, 0.999), eps=1e-8)
        off = 0
        for _ in range(case["iters"]):
            if off + case["batch"] > case["rows"]:
                off = 0
            rows = slice(off, off + case["batch"])
            loss = ((_forward(p, x[rows].double()) - t[rows].double()) ** 2).mean()
            opt.zero_grad()
            loss.backward()
            opt.step()
            off += case["batch"]
        return {"loss": float(loss.detach()), "params": p.detach()}
    fl = _flow(case)
    base = _base(fl)
    cons, u, v, w = _fields(case, fl, base, seed)
    if kind == "kessler":
        return [q for q in _kessler(fl.cfg, cons)]
    net = np.load(NET_FILE) if kind == "learned" else None
    cons, u, v, w = _Flat(fl.cfg, base).step(cons, u[:, :, :-1], v[:, :-1], w, net)
    return {"cons": [cons[n] for n in range(cons.shape[0])], "u": torch.cat([u, u[:, :, :1]], 2),
            "v": torch.cat([v, v[:, :1]], 1), "w": w}
