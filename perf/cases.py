"""Performance cases of the public entry points: what a user of this package
has the GPU do, from the smallest boxes to the 512^3 one.

Kinds of case
  solver    one box: `steps` time steps between two saves, then the save's
            download of rho, u and Q into pinned host buffers through the C
            ABI (the stepping loop of a simulation).
  driver    the same for the driver's default loop, which also writes a log
            line per save: flow and energy sums and the disclination lines.
  ensemble  many small boxes advanced together, then every box downloaded.
  gradient  loss and parameter gradients of the closure network (forward and
            backward) on one training pair.
  closure   corrected coarse steps: network and coarse solver step, then the
            download.
  analysis  the per-save diagnostics of one state: log sums, free energy,
            defect count, speed, velocity spectrum and Q correlation.

Saved fields are kept in the type of the box's precision after the float64
download: float64, float32, and float16 where the populations are stored in
FP16 (their rounding, 2^-11, is what such a box's fields carry).

`exact` restates the model in plain torch float64 (no code of this package).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import lbman3d_b200 as L
from lbman3d_b200 import _native as N
from lbman3d_b200.closure import Closure, coarse_params

PREC = {"fp64": L.Precision.FP64, "fp32": L.Precision.FP32, "fp16": L.Precision.FP16}
BC = {"periodic": L.FullyPeriodicConfig, "channel": L.ChannelConfig, "slit": L.SlitConfig,
      "slit_noslip": L.SlitNoSlipConfig}
STATE_BYTES = {"fp64": 368, "fp32": 184, "fp16": 124}  # f 15+15, Q 5+5, u 3+3 words per cell and step
STEP_FLOPS = 1100                                      # Q stage about 700, collision about 400 per cell


def listed():
    return [
        # The reference's smallest box (32^3, FP64): launches and latency.
        {"name": "periodic32_fp64", "kind": "solver", "nx": 32, "ny": 32, "nz": 32, "bc": "periodic",
         "precision": "fp64", "upwind": False, "alpha": 0.023, "steps": 1000},
        # The driver as it is started by default (20x100x100, FP64, no-slip
        # slit, a log line every 100 steps).
        {"name": "driver20_fp64", "kind": "driver", "nx": 20, "ny": 100, "nz": 100, "bc": "slit_noslip",
         "precision": "fp64", "upwind": False, "alpha": 0.023, "steps": 100},
        # Channel configuration, FP32, upwind advection.
        {"name": "channel20_fp32_upwind", "kind": "solver", "nx": 20, "ny": 100, "nz": 100, "bc": "channel",
         "precision": "fp32", "upwind": True, "alpha": 0.01, "steps": 200},
        # Odd sides in every direction (no tile or vector width divides them).
        {"name": "channel_odd_fp32", "kind": "solver", "nx": 67, "ny": 101, "nz": 131, "bc": "channel",
         "precision": "fp32", "upwind": False, "alpha": 0.02, "steps": 200},
        # Slit configuration, the production precision.
        {"name": "slit64_fp32", "kind": "solver", "nx": 64, "ny": 256, "nz": 256, "bc": "slit",
         "precision": "fp32", "upwind": False, "alpha": 0.01, "steps": 200},
        # The same box in the reference's arithmetic.
        {"name": "slit64_fp64", "kind": "solver", "nx": 64, "ny": 256, "nz": 256, "bc": "slit",
         "precision": "fp64", "upwind": False, "alpha": 0.01, "steps": 100},
        # Active turbulence, FP16 population storage.
        {"name": "periodic256_fp16", "kind": "solver", "nx": 256, "ny": 256, "nz": 256, "bc": "periodic",
         "precision": "fp16", "upwind": False, "alpha": 0.01, "steps": 200},
        # The headline box: 512^3, FP32, one save interval.
        {"name": "periodic512_fp32", "kind": "solver", "nx": 512, "ny": 512, "nz": 512, "bc": "periodic",
         "precision": "fp32", "upwind": False, "alpha": 0.01, "steps": 100},
        # A parameter scan: 96 boxes of sides 24..96, half periodic, half slit.
        {"name": "ensemble96_fp32", "kind": "ensemble", "boxes": 96, "mix": 2024, "precision": "fp32", "steps": 200},
        # Training the closure: one gradient on the 64^3 coarse grid.
        {"name": "closure_gradient64", "kind": "gradient", "nx": 64, "ny": 64, "nz": 64},
        # Using it: corrected coarse steps of the 64^3 grid.
        {"name": "closure_run64", "kind": "closure", "nx": 64, "ny": 64, "nz": 64, "steps": 100},
        # Diagnostics of a 256^3 state (statistics are taken at every save).
        {"name": "analysis256_fp32", "kind": "analysis", "nx": 256, "ny": 256, "nz": 256, "precision": "fp32"},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, lo, hi, least=8):
    """Sides of a box of about lo..hi cells, any integers, aspect ratios up to about 4."""
    s = _log_uniform(rng, lo, hi) ** (1.0 / 3.0)
    return [max(least, round(s * math.exp(rng.uniform(-0.5, 0.5)))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["solver"] * 5 + ["driver", "ensemble", "gradient", "closure", "analysis"])
    if kind == "solver":
        nx, ny, nz = _sides(rng, 2 ** 14, 2 ** 24.5)
        if rng.random() < 0.5:  # half of the boxes have the usual multiples of 4 along x
            nx = max(8, nx // 4 * 4)
        cells = nx * ny * nz
        return {"kind": "solver", "nx": nx, "ny": ny, "nz": nz, "bc": rng.choice(["periodic", "channel", "slit"]),
                "precision": rng.choice(["fp64", "fp32", "fp32", "fp16"]), "upwind": rng.random() < 0.3,
                "alpha": round(_log_uniform(rng, 0.005, 0.02), 4), "steps": int(max(60, min(200, 1.2e9 / cells)))}
    if kind == "driver":
        nx, ny, nz = _sides(rng, 2 ** 15, 2 ** 20)
        return {"kind": "driver", "nx": nx, "ny": ny, "nz": nz, "bc": rng.choice(["slit_noslip", "periodic", "channel"]),
                "precision": "fp64", "upwind": False, "alpha": round(_log_uniform(rng, 0.005, 0.02), 4), "steps": 100}
    if kind == "ensemble":
        return {"kind": "ensemble", "boxes": rng.randint(8, 96), "mix": rng.randint(1, 10 ** 6),
                "precision": rng.choice(["fp32", "fp32", "fp16", "fp64"]), "steps": 100}
    if kind == "analysis":
        nx, ny, nz = _sides(rng, 2 ** 17, 2 ** 24)
        return {"kind": "analysis", "nx": nx, "ny": ny, "nz": nz, "precision": rng.choice(["fp64", "fp32"])}
    side = lambda: 8 * rng.randint(3, 10)
    c = {"kind": kind, "nx": side(), "ny": 16 * rng.randint(2, 5) if rng.random() < 0.7 else side(), "nz": rng.randint(20, 80)}
    if kind == "closure":
        c["steps"] = rng.randint(20, 100)
    return c


# ---- inputs ---------------------------------------------------------------------
_DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=_DEV).manual_seed(seed & 0x7FFFFFFF)


def _director_q(V, S0, seed, sigma=1e-3):
    """Q of a uniformly random director per cell plus Gaussian noise: [5, V], float64, on the GPU."""
    g = _gen(seed)
    n = torch.randn(3, V, generator=g, device=_DEV, dtype=torch.float64)
    n /= n.norm(dim=0)
    q = torch.stack([n[0] * n[0] - 1 / 3, n[0] * n[1], n[0] * n[2], n[1] * n[1] - 1 / 3, n[1] * n[2]])
    return S0 * q + sigma * torch.randn(5, V, generator=g, device=_DEV, dtype=torch.float64)


def _smooth(count, nx, ny, nz, seed, cells=6.0):
    """`count` smooth periodic random fields of unit rms, correlation length about `cells`: [count, nz*ny*nx]."""
    g = _gen(seed)
    k2 = sum(torch.meshgrid(torch.fft.fftfreq(nz, device=_DEV) ** 2, torch.fft.fftfreq(ny, device=_DEV) ** 2,
                            torch.fft.rfftfreq(nx, device=_DEV) ** 2, indexing="ij"))
    filt = torch.exp(-0.5 * (2 * math.pi * cells) ** 2 * k2 / 4).double()
    out = torch.empty(count, nz * ny * nx, device=_DEV, dtype=torch.float64)
    for i in range(count):
        f = torch.fft.irfftn(torch.fft.rfftn(torch.randn(nz, ny, nx, generator=g, device=_DEV, dtype=torch.float64))
                             * filt, s=(nz, ny, nx)).reshape(-1)
        out[i] = f / f.square().mean().sqrt()
    return out


def _smooth_state(nx, ny, nz, seed):
    """(rho, u, Q) of a developed flow: smooth fields at the amplitudes of active turbulence."""
    s = _smooth(9, nx, ny, nz, seed)
    rho = 1.0 + 1e-3 * s[0]
    u = 0.02 * s[1:4] + torch.tensor([[3e-3], [-2e-3], [1e-3]], device=_DEV, dtype=torch.float64)
    q = 0.15 * s[4:9]
    return rho, u, q


def _params(case):
    return L.Params(nx=case["nx"], ny=case["ny"], nz=case["nz"], ALPHA=case["alpha"],
                    kQAdvection=L.Advection.Upwind if case["upwind"] else L.Advection.Centred)


_HOST = {}  # the pinned download buffers of the boxes in use, shared between handles of one size


def _host(name, n, dtype=torch.float64, pin=True):
    t = _HOST.get(name)
    if t is None or t.numel() != n or t.dtype != dtype:
        t = _HOST[name] = torch.empty(n, dtype=dtype, pin_memory=pin)
    return t


def _by_upload(case):
    return case["nx"] * case["ny"] * case["nz"] <= 2 ** 23


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solver", "driver"):
        p = _params(case)
        V = p.V
        sim = L.Simulation(p, BC[case["bc"]](), PREC[case["precision"]])
        if _by_upload(case):
            q = _director_q(V, L.EquilibriumScalarOrder(p), seed).cpu().numpy().reshape(-1)
            sim.upload(np.full(V, p.kDensity), np.zeros(3 * V), q)
        else:
            sim.init_seeded(seed, L.EquilibriumScalarOrder(p))
        return {"case": case, "sim": sim, "host": [_host(k, n * V) for k, n in (("rho", 1), ("u", 3), ("q", 5))]}
    if kind == "ensemble":
        boxes = L.draw_boxes(case["boxes"], seed=case["mix"])
        ens = L.Ensemble(boxes, PREC[case["precision"]])
        ens.init_seeded(seed)
        return {"case": case, "ens": ens, "boxes": boxes, "host": _host("ens", 9 * sum(p.V for p, _ in boxes))}
    if kind == "analysis":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        sim = L.Simulation(L.Params(nx=nx, ny=ny, nz=nz, ALPHA=0.01), L.FullyPeriodicConfig(), PREC[case["precision"]])
        rho, u, q = _smooth_state(nx, ny, nz, seed)
        sim.upload(rho.cpu().numpy(), u.cpu().numpy().reshape(-1), q.cpu().numpy().reshape(-1))
        return {"case": case, "sim": sim}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    V = nx * ny * nz
    c = Closure(nx, ny, nz, seed=1)
    c.set_params(_net_params(seed).float().numpy())
    c.set_scales(*[np.array(v, np.float32) for v in _SCALES])
    rho, u, q = _smooth_state(nx, ny, nz, seed)
    if kind == "gradient":
        x, t = _pair(case, seed)
        pin = lambda a: a.float().cpu().pin_memory().numpy()
        return {"case": case, "closure": c, "x": pin(x), "t": pin(t)}
    fine = L.Params(nx=4 * nx, ny=4 * ny, nz=4 * nz, ALPHA=0.01)
    coarse = L.Simulation(coarse_params(fine, 4), L.FullyPeriodicConfig(), L.Precision.FP32)
    coarse.upload(rho.cpu().numpy(), u.cpu().numpy().reshape(-1), q.cpu().numpy().reshape(-1))
    return {"case": case, "closure": c, "sim": coarse, "host": [_host(k, n * V) for k, n in (("rho", 1), ("u", 3), ("q", 5))]}


def _kept(name, host, precision):
    """The downloaded values in the type a save of this precision keeps."""
    if precision == "fp64":
        return host
    return _host(name + "_kept", host.numel(), torch.float32 if precision == "fp32" else torch.float16, False).copy_(host)


# ---- one pass -------------------------------------------------------------------
def _save(state, sim, precision):
    rho, u, q = state["host"]
    N.check(N.lib().lbman_download(sim.handle, N.dptr(rho.numpy()), N.dptr(u.numpy()), N.dptr(q.numpy()), None, None))
    return {k: _kept(k, v, precision) for k, v in (("rho", rho), ("u", u), ("q", q))}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solver":
        state["sim"].step(case["steps"])
        return _save(state, state["sim"], case["precision"])
    if kind == "driver":
        sim = state["sim"]
        for _ in range(case["steps"]):
            sim.step(1)
        out = _save(state, sim, case["precision"])
        d = sim.reduce(N.DIAG_FLOW | N.DIAG_ENERGY)
        info, _, _ = sim.defect_lines(with_points=False)
        return {**out, "log": [d["mass"], d["kinetic_energy"], d["free_energy"], d["umax2"]],
                "lines": [info["faces"], info["edges"], info["lines"]]}
    if kind == "ensemble":
        ens, host = state["ens"], state["host"]
        ens.step(case["steps"])
        h, at = host.numpy(), 0
        for b, (p, _) in enumerate(state["boxes"]):
            V = p.V
            N.check(N.lib().lbman_ensemble_download(ens._h, b, N.dptr(h[at:at + V]), N.dptr(h[at + V:at + 4 * V]),
                                                    N.dptr(h[at + 4 * V:at + 9 * V]), None))
            at += 9 * V
        return _kept("ens", host, case["precision"])
    if kind == "gradient":
        loss, g = state["closure"].gradient(state["x"], state["t"])
        return {"loss": loss, "grad": g}
    if kind == "closure":
        state["closure"].step(state["sim"], case["steps"])
        return _save(state, state["sim"], "fp32")
    sim = state["sim"]
    d = sim.reduce(N.DIAG_ALL)
    st = sim.statistics()
    E, nE = sim.velocity_spectrum()
    Cr, nC, xi = sim.q_correlation()
    return {"sums": [d["mass"], d["px"], d["py"], d["pz"], d["kinetic_energy"], d["umax2"], d["free_energy"]],
            "defect_faces": d["defect_faces"], "speed": [st["mean_speed"], st["rms_speed"]],
            "E": E, "nE": nE, "C": Cr, "nC": nC, "xi": xi}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(p.V for p, _ in L.draw_boxes(case["boxes"], seed=case["mix"]))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    if kind in ("solver", "driver", "ensemble"):
        n = cells * case["steps"]
        return {"bytes": n * STATE_BYTES[case["precision"]] + 72 * cells, "flops": n * STEP_FLOPS}
    mac = 27 * (9 * 32 + 32 * 32 + 32 * 32 + 32 * 8)  # the network, per cell
    if kind == "gradient":  # input, target, activations out and in; forward, backward data (not layer 1), weights
        return {"bytes": cells * (17 * 4 + 2 * 2 * 3 * 32), "flops": cells * 2 * (3 * mac - 27 * 9 * 32)}
    if kind == "closure":
        n = cells * case["steps"]
        return {"bytes": n * (STATE_BYTES["fp32"] + 9 * 4 + 8 * 4) + 72 * cells, "flops": n * (2 * mac + STEP_FLOPS)}
    w = 8 if case["precision"] == "fp64" else 4
    return {"bytes": cells * 9 * w, "flops": cells * 8 * 2.5 * math.log2(cells)}


# ---- the closure network --------------------------------------------------------
_LAYERS = ((16, 32, 9, 32), (32, 32, 32, 32), (32, 32, 32, 32), (32, 16, 32, 8))  # cin, cout, and those in use
_SCALES = ([1.0] + [0.0] * 8, [1e-3] + [0.02] * 3 + [0.15] * 5, [1e-3] * 5 + [1e-4] * 3)  # shift, scale, output scale


def _net_params(seed):
    """Weights [27, cin, cout] and biases of every layer, one flat float64 vector (on the host)."""
    g = torch.Generator().manual_seed(seed & 0x7FFFFFFF)
    out = []
    for i, (cin, cout, rin, rout) in enumerate(_LAYERS):
        w = torch.zeros(27, cin, cout, dtype=torch.float64)
        w[:, :rin, :rout] = torch.randn(27, rin, rout, generator=g, dtype=torch.float64) * math.sqrt(2 / (27 * rin)) * (0.1 if i == 3 else 1)
        b = torch.zeros(cout, dtype=torch.float64)
        b[:rout] = 0.05 * torch.randn(rout, generator=g, dtype=torch.float64)
        out += [w.reshape(-1), b]
    return torch.cat(out).float().double()


def _pair(case, seed):
    """A training pair: the state's 9 channels and the 8 corrections, as float32 holds them."""
    rho, u, q = _smooth_state(case["nx"], case["ny"], case["nz"], seed)
    t = _smooth(8, case["nx"], case["ny"], case["nz"], seed + 77) * torch.tensor(_SCALES[2], device=_DEV, dtype=torch.float64)[:, None]
    return torch.cat([rho[None], u, q]).float().double(), t.float().double()


def _network(p, x, nx, ny, nz):
    """Normalised outputs [8, V] of the network with parameters p for input channels x [9, V]."""
    shift, scale, _ = (torch.tensor(v, device=_DEV, dtype=torch.float64)[:, None] for v in _SCALES)
    a = ((x - shift) / scale).reshape(9, nz, ny, nx)
    at = 0
    for i, (cin, cout, rin, rout) in enumerate(_LAYERS):
        w = p[at:at + 27 * cin * cout].reshape(27, cin, cout)[:, :rin, :rout]
        at += 27 * cin * cout
        o = p[at:at + rout][:, None, None, None]
        at += cout
        for tap in range(27):  # output cell c reads c + (dx, dy, dz)
            d = (tap // 9 - 1, tap // 3 % 3 - 1, tap % 3 - 1)
            o = o + torch.einsum("izyx,io->ozyx", torch.roll(a, (-d[0], -d[1], -d[2]), (1, 2, 3)), w[tap])
        a = torch.nn.functional.gelu(o) if i < 3 else o
    return a.reshape(8, -1)


# ---- the solver, restated in float64 -----------------------------------------------
_E = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 1), (-1, 1, 1),
      (-1, -1, 1), (1, -1, 1), (1, 1, -1), (-1, 1, -1), (-1, -1, -1), (1, -1, -1)]
_W = [2 / 9] + [1 / 9] * 6 + [1 / 72] * 8
# walls per axis: None (periodic), "noslip" or "slip"; Q is Neumann on every wall
_WALLS = {"periodic": (None, None, None), "channel": ("noslip", "noslip", None), "slit": ("slip", None, None),
          "slit_noslip": ("noslip", None, None)}


class _Model:
    """Fields are [nz, ny, nx] float64; axis 0, 1, 2 = x, y, z."""

    def __init__(self, p, walls, upwind):
        self.p, self.walls, self.upwind = p, walls, upwind
        self.n = (p.nx, p.ny, p.nz)

    def at(self, a, ax, s, ghost=1.0):
        """The neighbour s = +-1 along ax; beyond a wall, `ghost` times the cell itself."""
        d = 2 - ax
        r = torch.roll(a, -s, d)
        if self.walls[ax]:
            i = self.n[ax] - 1 if s > 0 else 0
            r.select(d, i).copy_(ghost * a.select(d, i))
        return r

    def diff(self, a, ax, ghost=1.0):
        return 0.5 * (self.at(a, ax, 1, ghost) - self.at(a, ax, -1, ghost))

    def vgrad(self, u, c, ax):
        w = self.walls[ax]
        return self.diff(u, ax, -1.0 if w == "noslip" or (w == "slip" and c == ax) else 1.0)

    def full(self, q):
        return [[q[0], q[1], q[2]], [q[1], q[3], q[4]], [q[2], q[4], -(q[0] + q[3])]]

    def q_stage(self, q, u):
        """Q of the next step and the body force."""
        p, lam, I = self.p, self.p.LAMBDA, range(3)
        d = [[self.diff(c, ax) for ax in I] for c in q]
        d2 = [[self.at(c, ax, 1) + self.at(c, ax, -1) - 2 * c for ax in I] for c in q]
        adv = []
        for k in range(5):
            t = sum(u[ax] * d[k][ax] for ax in I)
            if self.upwind:
                t = t - sum(0.5 * u[ax].abs() * d2[k][ax] for ax in I)
            adv.append(t)
        Q = self.full(q)
        g = [[self.vgrad(u[c], c, ax) if not (c == 2 and ax == 2) else None for ax in I] for c in I]
        g[2][2] = -(g[0][0] + g[1][1])
        E = [[0.5 * (g[a][b] + g[b][a]) for b in I] for a in I]
        B = [[lam * E[a][b] - 0.5 * (g[a][b] - g[b][a]) for b in I] for a in I]
        mul = lambda X, Y: [[sum(X[a][k] * Y[k][b] for k in I) for b in I] for a in I]
        NB = mul(Q, B)
        T = NB[0][0] + NB[1][1] + NB[2][2]
        Q2 = mul(Q, Q)
        tr2 = Q2[0][0] + Q2[1][1] + Q2[2][2]
        idx = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2))
        h, qn = [], []
        for k, (a, b) in enumerate(idx):
            one = 1.0 if a == b else 0.0
            h.append(p.L * sum(d2[k]) - (p.A + p.C * tr2) * q[k] - p.B * (Q2[a][b] - one / 3 * tr2))
            rhs = -adv[k] + NB[a][b] + NB[b][a] - 2 / 3 * one * T - 2 * T * q[k] + lam * 2 / 3 * E[a][b]
            qn.append(q[k] + p.DT * (rhs + p.GAMMA * h[k]))
        H = self.full(h)
        dQ = [self.full([d[k][ax] for k in range(5)]) for ax in I]
        F = [-sum(H[a][b] * dQ[ax][a][b] for a in I for b in I) for ax in I]
        NH = mul(Q, H)
        tr = NH[0][0] + NH[1][1] + NH[2][2]
        Qn = self.full(qn)
        for a in I:
            for b in I:
                one = 1.0 if a == b else 0.0
                s = -2 / 3 * lam * H[a][b] - lam * (NH[a][b] + NH[b][a] - 2 / 3 * one * tr) + 2 * lam * tr * Q[a][b]
                F[a] = F[a] + self.diff(s + NH[a][b] - NH[b][a] - p.ALPHA * Qn[a][b], b)
            F[a] = F[a] - p.MU * u[a]
        return qn, F

    def feq(self, rho, u):
        u2 = sum(c * c for c in u)
        return [w * rho * (1 + 3 * s + 4.5 * s * s - 1.5 * u2)
                for w, s in ((w, sum(e * c for e, c in zip(ev, u))) for ev, w in zip(_E, _W))]

    def lbm(self, f, F):
        """Collide and stream: (rho, u) of the collision and the next populations."""
        p = self.p
        rho = sum(f)
        u = [(sum(ev[a] * c for ev, c in zip(_E, f) if ev[a]) + 0.5 * p.DT * F[a]) / rho for a in range(3)]
        uF = sum(a * b for a, b in zip(u, F))
        post = []
        for ev, w, fi, fe in zip(_E, _W, f, self.feq(rho, u)):
            ue, eF = (sum(e * c for e, c in zip(ev, v)) for v in (u, F))
            post.append(p.omega * fi + p.omega_prime * fe + p.DT * p.omega_forcing * w * (3 * eF - 3 * uF + 9 * ue * eF))
        nxt = []
        for j, ev in enumerate(_E):
            r = torch.roll(post[j], (ev[2], ev[1], ev[0]), (0, 1, 2))
            for ax in range(3):
                if self.walls[ax] and ev[ax]:
                    back = tuple(-e for e in ev) if self.walls[ax] == "noslip" else tuple(-e if k == ax else e for k, e in enumerate(ev))
                    i = 0 if ev[ax] > 0 else self.n[ax] - 1
                    r.select(2 - ax, i).copy_(post[_E.index(back)].select(2 - ax, i))
            nxt.append(r)
        return rho, u, nxt


def _exact_flow(case, seed, precision, steps):
    p = _params(case)
    m = _Model(p, _WALLS[case["bc"]], case["upwind"])
    shape = (p.nz, p.ny, p.nx)
    q = _director_q(p.V, L.EquilibriumScalarOrder(p), seed)
    if precision != "fp64":
        q = q.float().double()
    q = [c.reshape(shape) for c in q]
    rho = torch.full(shape, p.kDensity, device=_DEV, dtype=torch.float64)
    u = [torch.zeros_like(rho) for _ in range(3)]
    f = m.feq(rho, u)
    for _ in range(steps):
        q, F = m.q_stage(q, u)
        rho, u, f = m.lbm(f, F)
    flat = lambda v: torch.cat([c.reshape(-1) for c in v])
    return {"rho": rho.reshape(-1), "u": flat(u), "q": flat(q)}


def _exact_closure(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    p = coarse_params(L.Params(nx=4 * nx, ny=4 * ny, nz=4 * nz, ALPHA=0.01), 4)
    m = _Model(p, _WALLS["periodic"], False)
    par = _net_params(seed).to(_DEV)
    rho, u, q = (v.float().double() for v in _smooth_state(nx, ny, nz, seed))
    sc = torch.tensor(_SCALES[2], device=_DEV, dtype=torch.float64)[:, None]
    split = lambda v: [c.reshape(nz, ny, nx) for c in v]
    for _ in range(case["steps"]):
        corr = sc * _network(par, torch.cat([rho.reshape(1, -1), u, q]), nx, ny, nz)
        uu = split(u)
        qn, F = m.q_stage(split(q), uu)
        rho, un, _ = m.lbm(m.feq(rho.reshape(nz, ny, nx), uu), F)
        q = torch.stack([c.reshape(-1) for c in qn]) + corr[:5]
        u = torch.stack([c.reshape(-1) for c in un]) + corr[5:]
    return {"rho": rho.reshape(-1), "u": u.reshape(-1), "q": q.reshape(-1)}


def _exact_gradient(case, seed):
    par = _net_params(seed).to(_DEV).requires_grad_(True)
    x, t = _pair(case, seed)
    out = _network(par, x, case["nx"], case["ny"], case["nz"])
    sc = torch.tensor(_SCALES[2], device=_DEV, dtype=torch.float64)[:, None]
    loss = (out - t / sc).square().mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": par.grad}


def _shells(b, v, nbins):
    b, v = b.reshape(-1), v.reshape(-1)
    keep = b < nbins
    return torch.zeros(nbins, device=_DEV, dtype=torch.float64).index_add_(0, b[keep], v[keep])


def _exact_analysis(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    V, shape = nx * ny * nz, (nz, ny, nx)
    p = L.Params(nx=nx, ny=ny, nz=nz)
    rho, u, q = _smooth_state(nx, ny, nz, seed)
    if case["precision"] != "fp64":
        rho, u, q = (v.float().double() for v in (rho, u, q))
    u2 = u.square().sum(0)
    nbins = int(max(nx, ny, nz) * 3 ** 0.5 / 2) + 2
    m = _Model(p, _WALLS["periodic"], False)
    lap = [sum(m.at(c, ax, s) for ax in range(3) for s in (1, -1)) - 6 * c for c in (k.reshape(shape) for k in q)]
    Q, Lq = m.full(list(q)), m.full([c.reshape(-1) for c in lap])
    dot = lambda X, Y: sum(X[a][b] * Y[a][b] for a in range(3) for b in range(3))
    Q2 = [[sum(Q[a][k] * Q[k][b] for k in range(3)) for b in range(3)] for a in range(3)]
    tr2 = dot(Q, Q)
    energy = 0.5 * p.A * tr2 + p.B / 3 * dot(Q, Q2) + 0.25 * p.C * tr2 * tr2 - 0.5 * p.L * dot(Q, Lq)
    kz, ky, kx = torch.meshgrid(torch.fft.fftfreq(nz, device=_DEV, dtype=torch.float64), torch.fft.fftfreq(ny, device=_DEV, dtype=torch.float64),
                                torch.fft.fftfreq(nx, device=_DEV, dtype=torch.float64), indexing="ij")
    kb = (max(nx, ny, nz) * (kx * kx + ky * ky + kz * kz).sqrt() + 0.5).long()
    one = torch.ones(shape, device=_DEV, dtype=torch.float64)
    power = sum(torch.fft.fftn(c.reshape(shape)).abs().square() for c in u)
    E = 0.5 / V ** 2 * _shells(kb, power, nbins)
    qf = [torch.fft.fftn(c.reshape(shape)) for c in q]
    qp = dot(m.full(qf), [[c.conj() for c in r] for r in m.full(qf)]).real
    corr = torch.fft.ifftn(qp).real
    r = [torch.minimum(torch.arange(k, device=_DEV), k - torch.arange(k, device=_DEV)).double() for k in shape]
    rz, ry, rx = torch.meshgrid(*r, indexing="ij")
    rb = ((rx * rx + ry * ry + rz * rz).sqrt() + 0.5).long()
    nC = _shells(rb, one, nbins)
    C = torch.where(nC > 0, _shells(rb, corr, nbins) / nC.clamp(min=1), 0 * nC)
    C = C / C[0]
    mom = (rho * u).sum(1)
    return {"sums": [float(v) for v in (rho.sum(), *mom, 0.5 * (rho * u2).sum(), u2.max(), energy.sum())],
            "defect_faces": None, "speed": [float(u2.sqrt().mean()), float(u2.mean().sqrt())],
            "E": E, "nE": None, "C": C, "nC": None, "xi": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solver", "driver"):
        cells = case["nx"] * case["ny"] * case["nz"]
        if not _by_upload(case) or case["steps"] * (cells + 2 ** 18) > 2 ** 31:
            return None
        out = _exact_flow(case, seed, case["precision"], case["steps"])
        return out if kind == "solver" else {**out, "log": [None] * 4, "lines": [None] * 3}
    if kind == "closure":
        return _exact_closure(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "analysis":
        return _exact_analysis(case, seed)
    return None
