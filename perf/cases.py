"""The workloads whose speed this framework is held to.

Each case is one pass of what a program does with the public interface, once its cavities, batch or
network exist: advance a cavity by a number of iterations and read the fields back, run a batch of
cavities, predict steady fields with the warm-start network, train it by one step.

Sizes and parameters are those of the repository's own configurations (the 128^2 and 2048^2 squares and
the 128^3 cube of bench.py, the reference's 513^2 erf grid, the cavities of sweep_specs and
sample_cases, the network at batch 16 of 128^2 images), plus ragged ones.  A pass runs the tens to
hundreds of iterations that lie between two looks at a running simulation.

`exact` restates the lattice Boltzmann scheme and the network in 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from __graft_entry__ import load_package

lbm = load_package()

EPS = float(np.float32(1e-6))  # the stop criterion of the reference's loop


def listed():
    return [
        # a cavity small enough that a pass is launches and latency: a look at a toy problem every 20 iterations
        {"name": "cavity2d_48x40_f64", "kind": "cavity", "nx": 48, "ny": 40, "nz": 0, "Ra": 1e4, "Pr": 0.71,
         "grid": "tanh", "stretch": 1.5, "storage": "f64", "steps": 20},
        # the plain square cavity, a part of its run to the steady state (stop test on the device)
        {"name": "cavity2d_128_f64_run", "kind": "run", "nx": 128, "ny": 128, "nz": 0, "Ra": 1e4, "Pr": 0.71,
         "grid": "tanh", "stretch": 1.5, "storage": "f64", "steps": 500},
        # the grid and parameters the reference's own 2D program is compiled with
        {"name": "cavity2d_513_erf_f64", "kind": "cavity", "nx": 513, "ny": 513, "nz": 0, "Ra": 1e5, "Pr": 0.71,
         "grid": "erf", "stretch": 3.2, "storage": "f64", "steps": 200},
        # the large 2D cavity of the precision study, in the drop-in's precision
        {"name": "cavity2d_2048_f64", "kind": "cavity", "nx": 2048, "ny": 2048, "nz": 0, "Ra": 1e7, "Pr": 0.71,
         "grid": "tanh", "stretch": 1.5, "storage": "f64", "steps": 100},
        # FP32 storage on a ragged box, fields kept in single precision (how training fields are generated)
        {"name": "cavity2d_1023x771_f32", "kind": "cavity", "nx": 1023, "ny": 771, "nz": 0, "Ra": 1e6, "Pr": 1.7,
         "grid": "tanh", "stretch": 1.3, "storage": "f32", "steps": 200},
        # the cube of the headline benchmark
        {"name": "cavity3d_128_f64", "kind": "cavity", "nx": 128, "ny": 128, "nz": 128, "Ra": 1e5, "Pr": 0.71,
         "grid": "tanh", "stretch": 1.5, "storage": "f64", "steps": 100},
        # the same cube in FP32 storage
        {"name": "cavity3d_128_f32", "kind": "cavity", "nx": 128, "ny": 128, "nz": 128, "Ra": 1e5, "Pr": 0.71,
         "grid": "tanh", "stretch": 1.5, "storage": "f32", "steps": 150},
        # a small 3D box with no size a multiple of anything
        {"name": "cavity3d_61x50x47_f64", "kind": "cavity", "nx": 61, "ny": 50, "nz": 47, "Ra": 1e4, "Pr": 3.0,
         "grid": "tanh", "stretch": 1.5, "storage": "f64", "steps": 100},
        # a parameter sweep: cavities of uneven size advanced as one batch
        {"name": "batch_sweep32_f64", "kind": "batch", "n": 32, "sides": "sweep", "storage": "f64", "steps": 60},
        # the time-to-steady set: square cavities run as one batch with the stop test on the device
        {"name": "batch_steady16_f64", "kind": "steady", "n": 16, "sides": "square", "storage": "f64", "steps": 300,
         "every": 100},
        # one prediction of the warm-start network
        {"name": "predict_b1_r128", "kind": "predict", "B": 1, "R": 128},
        # one training step of the warm-start network
        {"name": "train_b16_r128", "kind": "train", "B": 16, "R": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    r = rng.random()
    phys = {"Ra": round(10 ** rng.uniform(3.0, 6.0), 1), "Pr": round(rng.uniform(0.71, 7.0), 3), "grid": "tanh",
            "stretch": round(rng.uniform(1.0, 2.0), 3)}
    storage = rng.choice(["f64", "f64", "f32"])
    if r < 0.40:
        # 2D: 40 nodes to 2048 along x, aspect 1/2 to 2
        nx = _log(rng, 40, 1900)
        ny = max(40, min(2048, int(nx * rng.uniform(0.5, 2.0))))
        if nx * ny > 2048 * 1900:
            ny = 2048 * 1900 // nx
        steps = max(20, min(400 if storage == "f64" else 200, int(8e10 / (240.0 * nx * ny))))
        steps = rng.randint(max(10, steps // 2), steps)
        return {"kind": rng.choice(["cavity", "cavity", "run"]) if storage == "f64" else "cavity", "nx": nx, "ny": ny,
                "nz": 0, **phys, "storage": storage, "steps": steps}
    if r < 0.65:
        # 3D: 20 nodes to 140 per axis
        n = _log(rng, 20, 120)
        nx, ny, nz = (max(16, min(140, int(n * rng.uniform(0.8, 1.2)))) for _ in range(3))
        steps = max(20, min(150, int(8e10 / (432.0 * nx * ny * nz))))
        steps = rng.randint(max(10, steps // 2), steps)
        return {"kind": "cavity", "nx": nx, "ny": ny, "nz": nz, **phys, "storage": storage, "steps": steps}
    if r < 0.75:
        return {"kind": "batch", "n": rng.randint(4, 24), "sides": "sweep", "storage": storage,
                "steps": rng.randint(20, 60)}
    if r < 0.82:
        return {"kind": "steady", "n": rng.randint(1, 20), "sides": "square", "storage": "f64",
                "steps": rng.choice([150, 200, 250]), "every": rng.choice([50, 70, 100])}
    if r < 0.90:
        # one 3x3 layer, forward and backward, of the network's channel counts
        cin, cout = rng.choice([(32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 256), (256, 256),
                                (384, 128), (192, 64), (96, 32)])
        h = _log(rng, 12, 128)
        b = max(1, min(16, int(4e9 / (h * h * cin * cout * 18))))
        return {"kind": "layer", "B": rng.randint(1, b), "H": h, "cin": cin, "cout": cout}
    R = 8 * rng.randint(2, 16)
    return {"kind": rng.choice(["predict", "train"]), "B": rng.randint(1, 16), "R": R}


# ---------------------------------------------------------------------------
# cavities
# ---------------------------------------------------------------------------
def _members(case, seed):
    """The cavities of a case: dicts of sizes and parameters (a batch's are drawn from a fixed seed)."""
    if "n" not in case:
        return [case]
    rng = np.random.default_rng(case["n"])
    out = []
    for _ in range(case["n"]):
        if case["sides"] == "sweep":
            nx = int(rng.choice([64, 96, 128, 192, 256, 384, 512]))
            ny = int(round(nx * rng.uniform(1.0, 4.0)))
        else:
            nx = ny = int(rng.choice([128, 160, 192, 224, 256]))
        out.append({"nx": nx, "ny": ny, "nz": 0, "Ra": float(10 ** rng.uniform(3.0, 6.0)),
                    "Pr": float(rng.uniform(0.71, 7.0)), "grid": "tanh", "stretch": float(rng.uniform(1.0, 2.0))})
    return out


def _fields(m, rng):
    """A developing flow: a conduction profile with a few smooth modes, weak smooth vortices, and temperature
    noise of amplitude 1e-4.  Arrays (ny, nx) or (nz, ny, nx)."""
    shape = ((m["nz"],) if m["nz"] else ()) + (m["ny"], m["nx"])
    axes = [(np.arange(n) + 0.5) / n for n in shape]

    def modes(amp):
        out = np.zeros(shape)
        for _ in range(2):
            term = amp * rng.uniform(0.5, 1.0) * rng.choice([-1.0, 1.0])
            for a, x in enumerate(axes):
                s = np.sin(math.pi * rng.integers(1, 4) * x)
                term = term * s.reshape([-1 if b == a else 1 for b in range(len(shape))])
            out += term
        return out

    heated = axes[-1] if len(shape) == 2 else axes[-2].reshape(1, -1, 1)
    T = 1.0 - heated + modes(0.05) + 1e-4 * rng.uniform(-1.0, 1.0, size=shape)
    u, v = modes(0.02), modes(0.02)
    w = modes(0.02) if len(shape) == 3 else None
    return {"rho": 1.0 + modes(1e-4), "u": u, "v": v, "w": w, "T": T}


def _coords(m):
    nz = m["nz"]
    if m["nx"] == m["ny"] and nz in (0, m["nx"]):
        return lbm.mesh(m["nx"], m["ny"], nz, m["grid"], m["stretch"])
    return lbm.mesh_box(m["nx"], m["ny"], nz, 1.0, m["ny"] / m["nx"], max(nz, 1) / m["nx"], m["grid"], m["stretch"])


def _keys(dim):
    return ("rho", "u", "v", "w", "T") if dim == 3 else ("rho", "u", "v", "T")


def _prepare_cavities(case, seed):
    ms = _members(case, seed)
    dim = 3 if ms[0]["nz"] else 2
    if "n" in case:
        batch = lbm.Batch(2, [{**m, "nz": 1, "coords": _coords(m)} for m in ms], storage=case["storage"])
        cavs = batch.members
    else:
        m, batch = ms[0], None
        cavs = [lbm.Cavity(dim, m["nx"], m["ny"], m["nz"] or 1, Ra=m["Ra"], Pr=m["Pr"], coords=_coords(m),
                           storage=case["storage"])]
    for i, (c, m) in enumerate(zip(cavs, ms)):
        f = _fields(m, np.random.default_rng([seed, i]))
        c.init_equilibrium(f["rho"], f["u"], f["v"], f["w"], f["T"])
    # pinned host arrays for the fields, as a program that reads them regularly keeps them; members one after another
    total = sum(c.nnode for c in cavs)
    host = {k: torch.empty(total, dtype=torch.float64, pin_memory=True) for k in _keys(dim)}
    views, at = [], 0
    for c in cavs:
        views.append({k: a[at:at + c.nnode].numpy() for k, a in host.items()})
        at += c.nnode
    return {"kind": case["kind"], "steps": case["steps"], "every": case.get("every"), "storage": case["storage"],
            "batch": batch, "cavs": cavs, "host": host, "views": views}


def _run_cavities(s):
    out = {}
    if s["kind"] == "cavity":
        s["cavs"][0].step(s["steps"])
        if s["storage"] == "f64":
            out["errU"], out["errT"] = s["cavs"][0].check()
    elif s["kind"] == "run":
        n, out["errU"], out["errT"] = s["cavs"][0].run(s["steps"], s["steps"], EPS)
        out["done"] = n
    elif s["kind"] == "batch":
        s["batch"].step(s["steps"])
        if s["storage"] == "f64":
            out["errU"], out["errT"] = s["batch"].check()
    else:
        out["status"], out["done"] = s["batch"].run_masked(None, s["steps"], s["every"], EPS)
    for c, v in zip(s["cavs"], s["views"]):
        c.get_macro_into(**v)
    for k, a in s["host"].items():
        # FP32 storage: its fields are single-precision numbers, kept as such
        out[k] = a if s["storage"] == "f64" else a.to(torch.float32)
    return out


# ---------------------------------------------------------------------------
# the warm-start network
# ---------------------------------------------------------------------------
LAYERS = [("e1a", 32, 32), ("e1b", 32, 32), ("e2a", 32, 64), ("e2b", 64, 64), ("e3a", 64, 128), ("e3b", 128, 128),
          ("ba", 128, 256), ("bb", 256, 256), ("d3a", 384, 128), ("d3b", 128, 128), ("d2a", 192, 64),
          ("d2b", 64, 64), ("d1a", 96, 32), ("d1b", 32, 32)]
LR = 1e-3


def _net_params(seed):
    """He-normal weights and small biases, as a network in training has."""
    rng = np.random.default_rng([seed, 1])
    p = {n: (rng.normal(0.0, math.sqrt(2.0 / (9 * ci)), size=(co, 9, ci)).astype(np.float32),
             rng.normal(0.0, 0.02, size=co).astype(np.float32)) for n, ci, co in LAYERS}
    p["head"] = (rng.normal(0.0, math.sqrt(1.0 / 32), size=(3, 32)).astype(np.float32),
                 rng.normal(0.0, 0.02, size=3).astype(np.float32))
    return p


def _net_inputs(B, R, seed):
    """The network's images: wall-clustered coordinate maps and the scaled Ra, Pr, stretch in the first five of
    32 channels; targets smooth and of unit size."""
    rng = np.random.default_rng([seed, 2])
    pix = (np.arange(R) + 0.5) / R
    x = np.zeros((B, R, R, 32), dtype=np.float32)
    t = np.zeros((B, R, R, 3), dtype=np.float32)
    for b in range(B):
        st = rng.uniform(1.0, 2.0)
        c = 0.5 * (np.tanh(st * (2.0 * pix - 1.0)) / np.tanh(st) + 1.0)
        x[b, ..., 0], x[b, ..., 1] = c[None, :], c[:, None]
        x[b, ..., 2:5] = rng.uniform(-1.0, 1.0, size=3)
        for j in range(3):
            k = rng.integers(1, 4, size=2)
            t[b, ..., j] = 2.0 * rng.uniform(-1.0, 1.0) * np.outer(np.sin(math.pi * k[0] * pix),
                                                                   np.sin(math.pi * k[1] * pix))
    return x, t.reshape(-1, 3)


def _layer_inputs(case, seed):
    """Activations, weights, saved pre-activations and incoming gradients of one layer, on `dev`-independent
    numpy arrays rounded to what the layer holds them in."""
    rng = np.random.default_rng([seed, 3])
    B, H, ci, co = case["B"], case["H"], case["cin"], case["cout"]
    f = lambda *s: rng.standard_normal(size=s, dtype=np.float32)  # noqa: E731
    x = torch.from_numpy(f(B, H, H, ci)).to(torch.bfloat16)
    w = (torch.from_numpy(f(co, 9, ci)) * math.sqrt(2.0 / (9 * ci))).to(torch.bfloat16)
    return {"x": x, "w": w, "b": torch.from_numpy(0.1 * f(co)), "z": torch.from_numpy(f(B, H, H, co)),
            "da": torch.from_numpy(f(B, H, H, co))}


def prepare(case, seed):
    if case["kind"] == "layer":
        s = {k: v.cuda() for k, v in _layer_inputs(case, seed).items()}
        B, H, ci, co = case["B"], case["H"], case["cin"], case["cout"]
        lib = lbm.surrogate.nn()
        P = B * H * H
        ws = max(lib.lbm_nn_wgrad_workspace(B, H, H, ci, co), lib.lbm_nn_colsum_workspace(P, co))
        f32 = {"dtype": torch.float32, "device": "cuda"}
        bf = {"dtype": torch.bfloat16, "device": "cuda"}
        s.update(kind="layer", lib=lib, dims=(B, H, ci, co), zo=torch.empty(B, H, H, co, **f32),
                 a=torch.empty(B, H, H, co, **bf), dz=torch.empty(B, H, H, co, **bf),
                 wt=torch.empty(ci, 9, co, **bf), dx=torch.empty(B, H, H, ci, **f32),
                 dw=torch.empty(co, 9, ci, **f32), db=torch.empty(co, **f32), ws=torch.empty(int(ws), **f32))
        return s
    if case["kind"] in ("predict", "train"):
        net = lbm.surrogate.Net(R=case["R"], params=_net_params(seed))
        net.buffers(case["B"])
        x, t = _net_inputs(case["B"], case["R"], seed)
        return {"kind": case["kind"], "net": net, "B": case["B"], "x": torch.from_numpy(x).cuda().to(torch.bfloat16),
                "t": torch.from_numpy(t).cuda()}
    return _prepare_cavities(case, seed)


def _run_layer(s):
    """One 3x3 layer's forward pass, then its backward pass from saved pre-activations and incoming gradients."""
    lib, (B, H, ci, co) = s["lib"], s["dims"]
    st = torch.cuda.current_stream().cuda_stream
    p = lambda k: s[k].data_ptr()  # noqa: E731
    P = B * H * H
    rc = [lib.lbm_nn_conv3x3(p("x"), ci, 0, p("w"), p("b"), B, H, H, ci, co, p("zo"), co, 0, 0, p("a"), co, 0, 1, st),
          lib.lbm_nn_silu_backward(p("da"), co, 0, p("z"), P, co, p("dz"), st),
          lib.lbm_nn_flip_weights(p("w"), p("wt"), co, ci, st),
          lib.lbm_nn_conv3x3_wgrad(p("dz"), p("x"), ci, 0, B, H, H, ci, co, p("ws"), s["ws"].numel(), p("dw"), st),
          lib.lbm_nn_colsum(p("dz"), P, co, p("ws"), p("db"), st),
          lib.lbm_nn_conv3x3(p("dz"), co, 0, p("wt"), None, B, H, H, co, ci, p("dx"), ci, 0, 0, None, 0, 0, 0, st)]
    if any(rc):
        raise RuntimeError(f"layer: status {rc}")
    return {"z": s["zo"], "a": s["a"], "dz": s["dz"], "dx": s["dx"], "dw": s["dw"], "db": s["db"]}


def run(state):
    kind = state["kind"]
    if kind == "layer":
        return _run_layer(state)
    if kind == "predict":
        # a bf16 network's prediction is good to bf16
        return {"y": state["net"].forward(state["x"]).to(torch.bfloat16)}
    if kind == "train":
        net, B = state["net"], state["B"]
        y = net.forward(state["x"])
        net.loss(state["t"], B)
        net.backward(B)
        net.adam(LR)
        return {"y": y.to(torch.bfloat16), "grad": net.grad.to(torch.bfloat16), "weights": net.pb}
    return _run_cavities(state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Cavities: each iteration reads and writes its state once (populations and carried force), the accounting of
    bench.py, and the fields leave once per pass; flops of the collision and the interpolation.  Network: the
    convolutions' multiply-adds, each layer's tensors read and written once, weights and optimiser state."""
    k = case["kind"]
    if k == "layer":
        P, ci, co = case["B"] * case["H"] ** 2, case["cin"], case["cout"]
        return {"bytes": P * (ci * (2 + 2 + 4) + co * (4 + 2 + 8 + 2)) + 9 * ci * co * 8, "flops": 54.0 * P * ci * co}
    if k in ("predict", "train"):
        R, B = case["R"], case["B"]
        res = {"e1": 1, "e2": 2, "e3": 4, "ba": 8, "bb": 8, "d3": 4, "d2": 2, "d1": 1}
        flops = bts = par = 0.0
        for n, ci, co in LAYERS:
            P = B * (R // res[n[:2]]) ** 2
            flops += 18.0 * P * ci * co
            bts += P * (2 * ci + 2 * co)
            par += 9 * ci * co + co
        if k == "predict":
            return {"bytes": bts + 2 * par + B * R * R * 12, "flops": flops}
        return {"bytes": 3 * bts + 30 * par + B * R * R * 36, "flops": 3 * flops}
    nodes = sum(m["nx"] * m["ny"] * max(1, m["nz"]) for m in _members(case, 0))
    three = bool(case.get("nz", 0))
    b = 8 if case["storage"] == "f64" else 4
    per = (2 * 26 + 2) * b if three else (2 * 14 + 2) * b
    return {"bytes": float(nodes) * (per * case["steps"] + 8 * (5 if three else 4)),
            "flops": float(nodes) * case["steps"] * (620 if three else 310)}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _axes(m):
    """Node coordinates with the walls' end points, the lattice unit and the time step, per axis in lattice units."""
    ns = [m["nx"], m["ny"]] + ([m["nz"]] if m["nz"] else [])
    square = len(set(ns)) == 1
    raw = []
    for n in ns:
        xi = np.arange(n + 2) / (n + 1)
        if m["grid"] == "erf":
            s = m["stretch"]
            c = np.array([0.5 * (math.erf(s * (v - 0.5)) / math.erf(0.5 * s) + 1.0) for v in xi])
        else:
            s = m["stretch"]
            c = 0.5 * (np.tanh(s * (2.0 * xi - 1.0)) / math.tanh(s) + 1.0)
        raw.append(c * (1.0 if square else n / ns[0]))
    dx0 = raw[0][1] - raw[0][0] if square else min(c[1] - c[0] for c in raw)
    L = 1.0 / dx0
    out = []
    for c in raw:
        c = c.copy()
        c[1:-1] -= dx0 / 2.0
        out.append(c * L)
    return out, L, dx0 * L


def _flow(dim):
    if dim == 2:
        e = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]
        et = e[:5]
    else:
        e = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
             (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1),
             (0, 1, -1), (0, -1, -1)]
        et = e[:7]
    return np.array(e, dtype=np.float64), np.array(et, dtype=np.float64)


def _moments(e, et):
    s = (e * e).sum(1)
    x, y = e[:, 0], e[:, 1]
    if e.shape[1] == 2:
        M = np.stack([1 + 0 * x, 3 * s - 4, 4.5 * s * s - 10.5 * s + 4, x, (3 * s - 5) * x, y, (3 * s - 5) * y,
                      x * x - y * y, x * y])
        st, a, b = (et * et).sum(1), et[:, 0], et[:, 1]
        N = np.stack([1 + 0 * a, a, b, st, a * a - b * b])
    else:
        z = e[:, 2]
        p, q = 3 * x * x - s, y * y - z * z
        M = np.stack([1 + 0 * x, 19 * s - 30, (21 * s * s - 53 * s + 24) / 2, x, (5 * s - 9) * x, y, (5 * s - 9) * y, z,
                      (5 * s - 9) * z, p, (3 * s - 5) * p, q, (3 * s - 5) * q, x * y, y * z, x * z,
                      (y * y - z * z) * x, (z * z - x * x) * y, (x * x - y * y) * z])
        st, a, b, c = (et * et).sum(1), et[:, 0], et[:, 1], et[:, 2]
        N = np.stack([1 + 0 * a, a, b, c, st, a * a - b * b, a * a - c * c])
    return M, N


class _Exact:
    """One cavity in 64 bits: interpolation-supplemented streaming, half-way walls, MRT collision."""

    def __init__(self, m, f):
        self.dev = _dev()
        T64 = lambda a: torch.as_tensor(a, dtype=torch.float64, device=self.dev)  # noqa: E731
        ax, L, self.dt = _axes(m)
        self.dim = len(ax)
        self.e, self.et = _flow(self.dim)
        M, N = _moments(self.e, self.et)
        self.M, self.N, self.Mi, self.Ni = T64(M), T64(N), T64(np.linalg.inv(M)), T64(np.linalg.inv(N))
        nu = 0.1 * (L - 1.0) * math.sqrt(m["Pr"]) / math.sqrt(3.0 * m["Ra"])
        self.gbeta = m["Ra"] * nu * (nu / m["Pr"]) / (L - 1.0) ** 3
        self.Snu = 1.0 / (3.0 * nu + 0.5)
        self.Sq = 8.0 * (2.0 - self.Snu) / (8.0 - self.Snu)
        k = 1.0 / self.Snu - 0.5
        self.sig = 1.0 / (0.5 + (4.0 * k / (3.0 * m["Pr"]) if self.dim == 2 else k / (0.5 * m["Pr"])))
        # interpolation weights per axis and shift, on the window of three nodes around (or nearest) each node
        self.w, self.ax = [], [self.dim - 1 - a for a in range(self.dim)]  # array axis of each coordinate axis
        for a, c in enumerate(ax):
            n = len(c) - 2
            lo = np.clip(np.arange(1, n + 1) - 1, 1, n - 2)
            per = {}
            for s in (1, -1):
                p = [c[lo + j] + s * self.dt for j in range(3)]
                x = c[1:-1]
                shape = [1] * self.dim
                shape[self.ax[a]] = n
                per[s] = [T64(((x - p[(j + 1) % 3]) * (x - p[(j + 2) % 3])
                               / ((p[j] - p[(j + 1) % 3]) * (p[j] - p[(j + 2) % 3]))).reshape(shape)) for j in range(3)]
            self.w.append(per)
        opp = lambda e: [int(np.nonzero((e == -v).all(1))[0][0]) for v in e]  # noqa: E731
        self.op, self.opt = opp(self.e), opp(self.et)
        self.heat = 0 if self.dim == 2 else 1
        self.wT = 0.125 if self.dim == 2 else 1.0 / 12.0
        # equilibrium of the initial fields, then the first collision
        w0 = [4 / 9, 1 / 9, 1 / 36] if self.dim == 2 else [1 / 3, 1 / 18, 1 / 36]
        self.rho, self.T = T64(f["rho"]), T64(f["T"])
        self.u = [T64(f[k]) for k in ("u", "v", "w")[:self.dim]]
        u2 = sum(c * c for c in self.u)
        fs, gs = [], []
        for v in self.e:
            un = sum(c * x for c, x in zip(self.u, v))
            fs.append(w0[int(abs(v).sum())] * self.rho * (1 + 3 * un + 4.5 * un * un - 1.5 * u2))
        for v in self.et:
            un = sum(c * x for c, x in zip(self.u, v))
            gs.append((0.5 if not v.any() else self.wT) * self.T * (1 + un * (4 if self.dim == 2 else 6)))
        self.prev = None
        self.f, self.g = torch.stack(fs), torch.stack(gs)
        self._collide()

    def _collide(self):
        rho, T, u, S, Sq, dt = self.rho, self.T, self.u, self.Snu, self.Sq, self.dt
        F = self.gbeta * T * rho
        m = torch.tensordot(self.M, self.f, 1)
        u2 = sum(c * c for c in u)
        zero = torch.zeros_like(rho)
        if self.dim == 2:
            x, y = u
            eq = [rho, rho * (3 * u2 - 2), rho * (1 - 3 * u2), rho * x, -rho * x, rho * y, -rho * y,
                  rho * (x * x - y * y), rho * x * y]
            src = [zero, (6 - 3 * S) * y * F, -(6 - 3 * S) * y * F, zero, zero, F, -(1 - 0.5 * Sq) * F,
                   -(2 - S) * y * F, (1 - 0.5 * S) * x * F]
            rate = [0, S, S, 0, Sq, 0, Sq, S, S]
        else:
            x, y, z = u
            e9, e11, h = rho * (3 * x * x - u2), rho * (y * y - z * z), 1 - 0.5 * S
            eq = [rho, rho * (19 * u2 - 11), rho * (3 - 5.5 * u2), rho * x, -2 / 3 * rho * x, rho * y,
                  -2 / 3 * rho * y, rho * z, -2 / 3 * rho * z, e9, -0.5 * e9, e11, -0.5 * e11, rho * x * y,
                  rho * y * z, rho * x * z, zero, zero, zero]
            src = [zero, (38 - 19 * S) * z * F, -(11 - 5.5 * S) * z * F, zero, zero, zero, zero, F,
                   -2 / 3 * (1 - 0.5 * Sq) * F, (S - 2) * z * F, h * z * F, -(2 - S) * z * F, h * z * F, zero,
                   h * y * F, h * x * F, zero, zero, zero]
            rate = [0, S, S, 0, Sq, 0, Sq, 0, Sq] + [S] * 7 + [Sq] * 3
        for a in range(len(rate)):
            m[a] += -rate[a] * (m[a] - eq[a]) + src[a] * dt
        self.f = torch.tensordot(self.Mi, m, 1)
        n = torch.tensordot(self.N, self.g, 1)
        d = self.dim
        k = 1.9 if d == 2 else 1.2
        eq = [T] + [T * c for c in u] + [0.5 * T] + [zero] * (d - 1)
        rate = [1.0] + [self.sig] * d + [k] * d
        for a in range(len(rate)):
            n[a] -= rate[a] * (n[a] - eq[a])
        self.g = torch.tensordot(self.Ni, n, 1)
        self.F = F

    def _shift(self, p, v):
        for a in range(self.dim):
            if v[a]:
                ax, n = self.ax[a], p.shape[self.ax[a]]
                cut = lambda i, j: p.narrow(ax, i, j - i)  # noqa: E731
                w = self.w[a][int(v[a])]
                p = (w[0] * torch.cat([cut(0, 1), cut(0, n - 2), cut(n - 3, n - 2)], ax)
                     + w[1] * torch.cat([cut(1, 2), cut(1, n - 1), cut(n - 2, n - 1)], ax)
                     + w[2] * torch.cat([cut(2, 3), cut(2, n), cut(n - 1, n)], ax))
        return p

    def step(self):
        f = torch.stack([self._shift(p, v) for p, v in zip(self.f, self.e)])
        g = torch.stack([self._shift(p, v) for p, v in zip(self.g, self.et)])
        for a in range(self.dim):
            for s in (1, -1):  # the wall the axis starts from sends populations along +a, the other along -a
                ix = 0 if s == 1 else -1
                for q, v in enumerate(self.e):
                    if v[a] == s:
                        f[q].select(self.ax[a], ix).copy_(self.f[self.op[q]].select(self.ax[a], ix))
                for q, v in enumerate(self.et):
                    if v[a] == s:
                        back = self.g[self.opt[q]].select(self.ax[a], ix)
                        if a == self.heat:
                            back = -back + 2.0 * self.wT * (1.0 if s == 1 else 0.0)
                        g[q].select(self.ax[a], ix).copy_(back)
        self.f, self.g = f, g
        self.rho, self.T = f.sum(0), g.sum(0)
        mom = torch.tensordot(torch.as_tensor(self.e.T.copy(), device=self.dev), f, 1)
        mom[self.dim - 1] += 0.5 * self.dt * self.F
        self.u = [c / self.rho for c in mom]
        self._collide()

    def check(self):
        """Residuals against the fields of the previous check (zero before the first)."""
        now = self.u + [self.T]
        old = self.prev or [torch.zeros_like(self.T)] * len(now)
        self.prev = now
        n = lambda v: math.sqrt(sum(float((c * c).sum()) for c in v))  # noqa: E731
        d = [p - q for p, q in zip(now, old)]
        return n(d[:-1]) / n(now[:-1]), n(d[-1:]) / n(now[-1:])


def _exact_cavities(case, seed):
    ms = _members(case, seed)
    dim = 3 if ms[0]["nz"] else 2
    fields = {k: [] for k in _keys(dim)}
    eu, et = [], []
    for i, m in enumerate(ms):
        x = _Exact(m, _fields(m, np.random.default_rng([seed, i])))
        for _ in range(case["steps"]):
            x.step()
        a, b = x.check()
        eu.append(a)
        et.append(b)
        vals = {"rho": x.rho, "T": x.T, **dict(zip(("u", "v", "w"), x.u))}
        for k in fields:
            fields[k].append(vals[k].reshape(-1).cpu())
    out = {k: torch.cat(v) for k, v in fields.items()}
    if case["kind"] == "steady":
        return {**out, "status": None, "done": None}
    if case["storage"] == "f64":
        out["errU"], out["errT"] = (np.array(eu), np.array(et)) if "n" in case else (eu[0], et[0])
    if case["kind"] == "run":
        out["done"] = None
    return out


def _conv(x, w):
    """x (B, H, W, Cin), w (Cout, 9, Cin) -> (B, H, W, Cout), zero padding of one."""
    k = w.reshape(w.shape[0], 3, 3, -1).permute(0, 3, 1, 2)
    return torch.nn.functional.conv2d(x.permute(0, 3, 1, 2), k, padding=1).permute(0, 2, 3, 1)


def _exact_net(case, seed):
    dev = _dev()
    B, R = case["B"], case["R"]
    x, t = _net_inputs(B, R, seed)
    x = torch.from_numpy(x).to(torch.bfloat16).double().to(dev)
    p = {}
    for k, (w, b) in _net_params(seed).items():
        w = torch.from_numpy(w)
        p[k] = [w.to(torch.bfloat16).double().to(dev).requires_grad_(), torch.from_numpy(b).double().to(dev).requires_grad_()]
    silu = torch.nn.functional.silu

    def layer(n, v):
        return silu(_conv(v, p[n][0]) + p[n][1])

    def pool(v):
        return torch.nn.functional.avg_pool2d(v.permute(0, 3, 1, 2), 2).permute(0, 2, 3, 1)

    def up(v):
        return v.repeat_interleave(2, 1).repeat_interleave(2, 2)

    with torch.set_grad_enabled(case["kind"] == "train"):
        s1 = layer("e1b", layer("e1a", x))
        s2 = layer("e2b", layer("e2a", pool(s1)))
        s3 = layer("e3b", layer("e3a", pool(s2)))
        v = layer("bb", layer("ba", pool(s3)))
        v = layer("d3b", layer("d3a", torch.cat([up(v), s3], -1)))
        v = layer("d2b", layer("d2a", torch.cat([up(v), s2], -1)))
        v = layer("d1b", layer("d1a", torch.cat([up(v), s1], -1)))
        y = (v @ p["head"][0].T + p["head"][1]).reshape(-1, 3)
        if case["kind"] == "predict":
            return {"y": y}
        loss = ((y - torch.from_numpy(t).double().to(dev)) ** 2).mean()
        loss.backward()
    # the flat parameter vector: each layer's weights and bias start at multiples of 64
    al = lambda n: (n + 63) // 64 * 64  # noqa: E731
    parts = {}
    at = 0
    for n, ci, co in LAYERS + [("head", 32, 3)]:
        size = 9 * ci * co if n != "head" else 96
        parts[n] = (at, al(at + size))
        at = al(parts[n][1] + co)
    grad, weights = torch.zeros(at, dtype=torch.float64, device=dev), torch.zeros(at, dtype=torch.float64, device=dev)
    master = _net_params(seed)
    for n, (ow, ob) in parts.items():
        for k, o in ((0, ow), (1, ob)):
            g = p[n][k].grad.reshape(-1)
            grad[o:o + g.numel()] = g
            w = torch.from_numpy(master[n][k]).double().to(dev).reshape(-1)
            # first Adam step: m / c1 = g, sqrt(v / c2) = |g|
            weights[o:o + g.numel()] = w - LR * g / (g.abs() + 1e-8)
    return {"y": y.detach(), "grad": grad, "weights": weights}


def exact(case, seed):
    if case["kind"] == "layer":
        s = {k: v.double().to(_dev()) for k, v in _layer_inputs(case, seed).items()}
        z = _conv(s["x"], s["w"]) + s["b"]
        sg = torch.sigmoid(s["z"])
        full = s["da"] * sg * (1 + s["z"] * (1 - sg))
        dz = full.to(torch.float32).to(torch.bfloat16).double()  # gradients enter the products in bf16
        w, x = s["w"].clone().requires_grad_(), s["x"].clone().requires_grad_()
        _conv(x, w).backward(dz)
        return {"z": z, "a": z * torch.sigmoid(z), "dz": full, "dx": x.grad, "dw": w.grad,
                "db": dz.sum((0, 1, 2))}
    if case["kind"] in ("predict", "train"):
        return _exact_net(case, seed)
    return _exact_cavities(case, seed)
