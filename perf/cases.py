"""Performance cases: the work a user of this package has it do, through its public entry points.

A case is a dict of plain values.  Its "kind" names the call:

  step     a two-phase jet (or periodic box) advanced by a number of steps, as a captured graph or as
           single calls, with the macroscopic fields of the last step and the running means as options;
           the state after the steps (both population sets) comes back
  sweep    many small jets advanced together (``batch.Sweep``)
  closure  a coarse lattice run with the learned closure: refresh, then steps
  train    Adam steps of the closure network on random mini-batches
  data     a fine snapshot turned into training data (filter, targets, features) and predicted on
  monitor  a snapshot's statistics: global reductions, phase-field flux, centreline, droplets

Inputs come from the seed alone: a liquid column on the inlet, small drops and a smooth velocity field.
``exact`` restates every path with torch in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

from ssmdlbm_b200 import _lib, batch, closure, configs
from ssmdlbm_b200._lib import check, lib
from ssmdlbm_b200.lbm import Simulation

STORAGE = {"f32": _lib.STORAGE_F32, "f16": _lib.STORAGE_F16, "bf16": _lib.STORAGE_BF16, "f16g32": _lib.STORAGE_F16_G32}
SIZES = {"f32": (4, 4), "f16": (2, 2), "bf16": (2, 2), "f16g32": (2, 4)}  # bytes of one f, one g
FLOPS = {19: 420, 27: 553}  # FP32 operations of one cell update
NET_SCALE, NET_OFFSET = (2e-3, 0.2), (1e-3, 1.0)
NUT_MAX = 0.02


# ------------------------------------------------------------------ the cases
def _step(name, nx, ny, nz, q, storage, steps, bc="jet", graph=True, store=False, means=False):
    return {"name": name, "kind": "step", "bc": bc, "nx": nx, "ny": ny, "nz": nz, "q": q, "storage": storage,
            "steps": steps, "graph": graph, "store": store, "means": means}


def listed():
    return [
        # a first look at a configuration on a small lattice: launch latency and idle SMs count
        _step("jet_q19_f32_64", 64, 64, 128, 19, "f32", 20),
        # the benchmark jet, and the same in half precision
        _step("jet_q27_f32_128", 128, 128, 512, 27, "f32", 10),
        _step("jet_q27_f16_128", 128, 128, 512, 27, "f16", 10),
        # the fine run of a closure study: a production lattice
        _step("jet_q19_f32_256", 256, 256, 1024, 19, "f32", 2),
        # the two-jet crossflow with ghost layers on every face, odd sizes, the reference's half layout,
        # single calls, the last step saved
        _step("cross_q27_f16g32_odd", 101, 75, 203, 27, "f16g32", 10, bc="cross", graph=False, store=True),
        # a closed periodic box of odd sizes: a unit test or a relaxation study
        _step("box_q19_bf16_odd", 67, 45, 51, 19, "bf16", 10, bc="box", graph=False),
        # time averages taken along a run, vorticity of the last step
        _step("means_q19_f32_96", 96, 96, 192, 19, "f32", 10, graph=False, store=True, means=True),
        # a parameter sweep of uneven jets
        {"name": "sweep_q19_f32_24", "kind": "sweep", "count": 24, "set": 2, "q": 19, "storage": "f32", "steps": 4},
        # a coarse production run with the closure: one refresh and the steps up to the next
        {"name": "closure_q27_f16_96", "kind": "closure", "nx": 96, "ny": 96, "nz": 384, "q": 27, "storage": "f16",
         "steps": 10},
        # the closure network's training loop at its default batch
        {"name": "train_64k", "kind": "train", "rows": 1000000, "batch": 65536, "steps": 10},
        # one fine snapshot into training data, and the network's prediction on it
        {"name": "data_128", "kind": "data", "nx": 128, "ny": 128, "nz": 512},
        # a snapshot's statistics
        {"name": "monitor_128", "kind": "monitor", "nx": 128, "ny": 128, "nz": 512, "storage": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axes(rng, most, even=False):
    """Sizes of a lattice of up to `most` cells, longer along z."""
    while True:
        nx = _log(rng, 24, 200)
        ny = nx if rng.random() < 0.4 else _log(rng, 20, 160)
        nz = int(nx * rng.choice((1, 2, 4))) + rng.choice((0, 0, 1, 3))
        if even:
            nx, ny, nz = 2 * (nx // 2), 2 * (ny // 2), 2 * (nz // 2)
        if 32 <= nz <= 800 and nx * ny * nz <= most:
            return nx, ny, nz


def draw(rng):
    kind = rng.choice(("step",) * 7 + ("sweep", "closure", "train", "data", "monitor"))
    q, storage = rng.choice((19, 27)), rng.choice(("f32", "f32", "f16", "bf16", "f16g32"))
    if kind == "step":
        nx, ny, nz = _axes(rng, 12_000_000)
        bc = rng.choice(("jet", "jet", "cross", "box"))
        graph = rng.random() < 0.5
        means = not graph and rng.random() < 0.3
        c = _step("", nx, ny, nz, q, storage, 2 * _log(rng, 1, 10), bc, graph, not graph and (means or rng.random() < 0.5),
                  means)
        while c["steps"] > 2 and nx * ny * nz * c["steps"] > 100_000_000:
            c["steps"] -= 2
        del c["name"]
        return c
    if kind == "sweep":
        return {"kind": kind, "count": _log(rng, 4, 24), "set": rng.randrange(1000), "q": q,
                "storage": rng.choice(("f32", "f16", "bf16")), "steps": 2 * rng.randrange(1, 3)}
    if kind == "closure":
        nx, ny, nz = _axes(rng, 4_000_000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "q": q, "storage": storage, "steps": rng.choice((1, 5, 10))}
    if kind == "train":
        return {"kind": kind, "rows": _log(rng, 200_000, 2_000_000), "batch": _log(rng, 2000, 120_000), "steps": rng.randrange(2, 11)}
    nx, ny, nz = _axes(rng, 8_000_000, even=kind == "data")
    if kind == "data":
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "storage": storage}


# ------------------------------------------------------------------ inputs
def _jet_values(c):
    """The physical parameters of a jet or box case, in lattice units."""
    return {"tau": 0.55, "sigma": 1e-3, "width": 4.0, "mobility": 0.1, "w_in": 0.05, "noise": 0.01,
            "diam": max(6, min(c["nx"], c["ny"]) // 8)}


def _params(c, seed):
    bc = c.get("bc", "jet")
    if bc == "cross":
        d = max(6, min(c["nx"], c["ny"]) // 8)
        p = configs.reference_like(c["nx"], c["ny"], c["nz"], c["q"], u_water=0.05, u_oil=0.05, diam_water=d, diam_oil=d,
                                   reynolds_water=3.0 * d, reynolds_oil=2.5 * d, weber=2.5 * d, interface_width=4.0)
        p.storage = STORAGE[c["storage"]]
        return p
    v = _jet_values(c)
    if bc == "box":
        return configs.periodic_box((c["nx"], c["ny"], c["nz"]), c["q"], tau=v["tau"], sigma=v["sigma"], width=v["width"],
                                    mobility=v["mobility"], storage=STORAGE[c["storage"]])
    return configs.oil_jet(c["nx"], c["ny"], c["nz"], c.get("q", 19), seed=seed, storage=STORAGE[c.get("storage", "f32")], **v)


def _fields(shape, seed, bc="jet", w_in=0.05, diam=8):
    """rho, ux, uy, uz, phi of a jet under way, float32 [z][y][x] on the GPU: a liquid column on the inlet's
    axis up to a third of the lattice, drops of radius 2-4 cells with phi cut to 0 below 1e-6, a smooth
    velocity field of amplitude 0.02, and the inlet face."""
    nz, ny, nx = shape
    dev = torch.device("cuda")
    rng = np.random.default_rng(seed)

    def wave(n):
        return np.sin(2 * np.pi * rng.integers(1, 4) * np.arange(n) / n + rng.uniform(0, 2 * np.pi))

    def smooth(scale):
        a, b, c = (torch.as_tensor(wave(n), device=dev) for n in (nz, ny, nx))
        return (scale * a[:, None, None] * b[None, :, None] * c[None, None, :]).float()

    ux, uy, uz, rho = smooth(0.02), smooth(0.02), smooth(0.02), 1.0 + smooth(1e-3)
    phi = torch.zeros(nz * ny * nx, device=dev)
    h = 8
    count = max(3, int(12e-6 * nx * ny * nz))
    size = np.array([nz, ny, nx])
    at = rng.uniform(h, np.maximum(size - h - 1, h + 1), (count, 3))
    rad = rng.uniform(2.0, 4.0, count)
    k = torch.arange(-h, h + 1, device=dev, dtype=torch.float64)
    base = np.floor(at)
    off = torch.as_tensor(base - at, device=dev)
    first = torch.as_tensor(base.astype(np.int64), device=dev)
    for s in range(0, count, 64):
        o, f = off[s:s + 64], first[s:s + 64]
        d2 = ((k[None, :, None, None] + o[:, 0, None, None, None]) ** 2 + (k[None, None, :, None] + o[:, 1, None, None, None]) ** 2
              + (k[None, None, None, :] + o[:, 2, None, None, None]) ** 2)
        v = 0.5 * (1.0 - torch.tanh(0.5 * (d2.sqrt() - torch.as_tensor(rad[s:s + 64], device=dev)[:, None, None, None])))
        v[v < 1e-6] = 0.0
        kk = k.long()
        z, y, x = ((kk[None] + f[:, d, None]) % int(size[d]) for d in range(3))
        i = (z[:, :, None, None] * ny + y[:, None, :, None]) * nx + x[:, None, None, :]
        phi.scatter_reduce_(0, i.reshape(-1), v.float().reshape(-1), "amax")
    phi = phi.reshape(shape)
    cy, cx = (ny - 1) * (0.25 if bc == "cross" else 0.5), (nx - 1) * 0.5
    y, x = (torch.arange(n, device=dev, dtype=torch.float64) for n in (ny, nx))
    r = ((y[:, None] - cy) ** 2 + (x[None, :] - cx) ** 2).sqrt()
    if bc != "box":
        column = 0.5 * (1.0 - torch.tanh(0.5 * (r - 0.5 * diam)))
        z = torch.arange(nz, device=dev, dtype=torch.float64)
        column = column[None] * (0.5 * (1.0 - torch.tanh(0.5 * (z - nz / 3.0))))[:, None, None]
        column[column < 1e-6] = 0.0
        phi = torch.maximum(phi, column.float())
        uz += w_in * phi
        disc = (r <= diam // 2)
        phi[0] = disc.float()
        uz[0] = w_in * disc.float()
        phi[-1] = 0.0
    return rho, ux, uy, uz, phi


def _start(sim, fields):
    """A lattice at equilibrium of the given macroscopic fields."""
    with torch.cuda.stream(sim.torch_stream):
        sim.torch_stream.wait_stream(torch.cuda.default_stream())
        for k, v in zip(("rho", "ux", "uy", "uz", "phi"), fields):
            sim.t[k].copy_(v.reshape(-1))
    check(lib().ssmd_init_from_macros(ctypes.byref(sim.p), ctypes.byref(sim.fields), sim.stream))
    sim.steps_done = 0
    sim.sync()


def _diam(c):
    return _jet_values(c)["diam"]


def _net_values(seed):
    """Weights and normalisation of a closure network (the layout of SSMD_MLP_NET_FLOATS)."""
    rng = np.random.default_rng(1000 + seed)
    w1 = np.zeros((64, 16))
    w1[:, :12] = rng.normal(0, 12 ** -0.5, (64, 12))
    parts = [w1.ravel(), rng.normal(0, 0.1, 64), rng.normal(0, 0.125, 4096), rng.normal(0, 0.1, 64),
             rng.normal(0, 0.125, 128), rng.normal(0, 0.1, 2), FEATURE_MEAN, 1.0 / FEATURE_STD, NET_SCALE, NET_OFFSET]
    return np.concatenate([np.asarray(v, np.float64) for v in parts]).astype(np.float32)


# what the twelve features of such fields are about
FEATURE_MEAN = np.array([0.02, 0.02, 0.01, 0.0, 2e-3, 2e-3, 0.0, 0.02, 2e-3, 0.0, 0.0, 0.0167])
FEATURE_STD = np.array([0.1, 0.1, 0.03, 0.05, 3e-3, 3e-3, 2e-3, 0.02, 0.02, 1e-3, 2e-3, 1e-3])


def _rows(c, seed):
    """Training rows: standardised features around their means, targets that follow them, weights."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(c["rows"], 12, device="cuda", generator=g)
    t = torch.stack((torch.tanh(x[:, 0] + 0.5 * x[:, 4]), x[:, 2] * torch.sigmoid(x[:, 3])), 1)
    t += 0.1 * torch.randn(c["rows"], 2, device="cuda", generator=g)
    mean, std = (torch.tensor(v, device="cuda", dtype=torch.float32) for v in (FEATURE_MEAN, FEATURE_STD))
    scale, offset = (torch.tensor(v, device="cuda") for v in (NET_SCALE, NET_OFFSET))
    w = torch.rand(c["rows"], 2, device="cuda", generator=g) + 0.01
    return x * std + mean, t * scale + offset, w


# ------------------------------------------------------------------ what a program has in hand
def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind == "train":
        net = closure.Network(0)
        net.net.copy_(torch.as_tensor(_net_values(seed)))
        s["net"], s["rows"] = net, _rows(c, seed)
        return s
    if kind == "sweep":
        sw = batch.Sweep(batch.sweep_params(c["count"], c["set"], c["q"], STORAGE[c["storage"]]), tile_z=32)
        for i, sim in enumerate(sw.sims):
            w, d = float(sim.p.u_oil), int(2 * round(math.sqrt(float(sim.p.oil_r2))))
            _start(sim, _fields(sim.shape, 1000 * seed + i, "jet", w, max(d, 4)))
        sw.run_graph(0, 2)  # captured once, replayed by every pass
        s["sweep"] = sw
        return s
    sim = Simulation(_params(c, seed))
    s["sim"] = sim
    _start(sim, _fields(sim.shape, seed, c.get("bc", "jet"), 0.05, _diam(c)))
    if kind in ("closure", "data"):
        net = closure.Network(0)
        net.net.copy_(torch.as_tensor(_net_values(seed)))
        s["net"] = net
    if kind == "closure":
        s["nut"], s["cs"] = torch.zeros(sim.cells, device="cuda"), torch.ones(sim.cells, device="cuda")
        s["arrays"] = _lib.Closure(s["nut"].data_ptr(), s["cs"].data_ptr())
        sim.p.closure = ctypes.addressof(s["arrays"])
    if kind == "data":
        cp = closure.coarse_params(sim.p)
        n = sim.cells // 8
        s["cp"] = cp
        s["coarse"], s["tau"], s["area"] = (torch.empty(k * n, device="cuda") for k in (5, 6, 1))
        s["feats"], s["targets"], s["weights"] = (torch.empty(n, k, device="cuda") for k in (12, 2, 2))
        s["view"] = closure._view(s["coarse"], n)
    if kind == "step":
        if c["means"]:
            sim.enable_derived()
        if c["graph"]:
            sim.graph(2)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def _now(sim):
    """The populations of the lattice's current parity."""
    a = sim.steps_done % 2 == 0
    return {"f": sim.t["f" if a else "f_alt"], "g": sim.t["g" if a else "g_alt"]}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "train":
        net = state["net"]
        net.train(*state["rows"], steps=c["steps"], batch=c["batch"], lr=1e-3, seed=1, average=0.9999)
        return {"net": net.net, "grad": net.grad, "m": net.m, "v": net.v, "loss": net.loss}
    if kind == "sweep":
        state["sweep"].run_graph(c["steps"] // 2, 2)
        return [_now(sim) for sim in state["sweep"].sims]
    sim = state["sim"]
    if kind == "step":
        if c["graph"]:
            sim.run_graph(c["steps"] // 2, 2)
        else:
            sim.step(c["steps"], store_macros=c["store"], average=c["means"])
        out = _now(sim)
        if c["store"]:
            out |= {k: sim.t[k] for k in ("rho", "ux", "uy", "uz", "phi")}
        if c["means"]:
            sim.derived_update(_lib.DERIVED_VORTICITY)
            out |= {k: sim.t[k] for k in sim.DERIVED}
        return out
    if kind == "closure":
        check(lib().ssmd_closure_refresh(ctypes.byref(sim.p), ctypes.byref(sim.fields), state["net"].net.data_ptr(), NUT_MAX,
                                         state["nut"].data_ptr(), state["cs"].data_ptr(), sim.stream))
        sim.step(c["steps"], store_macros=True)
        return _now(sim) | {k: sim.t[k] for k in ("rho", "ux", "uy", "uz", "phi")} | {"nut": state["nut"], "cs": state["cs"]}
    if kind == "data":
        s, L, st = state, lib(), sim.stream
        check(L.ssmd_closure_filter(ctypes.byref(sim.p), ctypes.byref(sim.fields), s["coarse"].data_ptr(), s["tau"].data_ptr(),
                                    s["area"].data_ptr(), st))
        check(L.ssmd_closure_targets(ctypes.byref(s["cp"]), s["coarse"].data_ptr(), s["tau"].data_ptr(), s["area"].data_ptr(),
                                     NUT_MAX, s["targets"].data_ptr(), s["weights"].data_ptr(), st))
        check(L.ssmd_closure_features(ctypes.byref(s["cp"]), ctypes.byref(s["view"]), s["feats"].data_ptr(), st))
        with torch.cuda.stream(sim.torch_stream):
            out = s["net"].predict(s["feats"])
        out.record_stream(torch.cuda.default_stream())
        return {k: s[k] for k in ("coarse", "tau", "area", "targets", "weights", "feats")} | {"predicted": out}
    st = sim.reduce()
    uz, phi = sim.centreline()
    drops = sim.droplets(0.5)
    return {"sums": np.array([st["phi_sum"], st["phi_sum_next"], st["mass"], *st["momentum"], st["kinetic"], st["u_max"],
                              st["nonfinite"], st["cells"]]),
            "flux": np.array(sim.phase_flux()), "uz": uz, "phi": phi,
            "root": _padded(drops["root"].astype(np.int64)), "cells": _padded(drops["cells"].astype(np.int64)),
            "volume": _padded(drops["volume"]), "inlet": _padded(drops["touches_inlet"].astype(np.int64))}


def _padded(a, size=1024):
    """A droplet list in an array of one length for every snapshot (their numbers differ)."""
    out = np.zeros(size, a.dtype)
    out[:len(a)] = a
    return out


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        return {"bytes": c["steps"] * c["batch"] * 64, "flops": c["steps"] * c["batch"] * 6 * (12 * 64 + 64 * 64 + 64 * 2)}
    if kind == "sweep":
        cells = sum(int(p.nx) * int(p.ny) * int(p.nz) for p in batch.sweep_params(c["count"], c["set"], c["q"]))
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
    if kind == "data":
        return {"bytes": cells * 20 + cells // 8 * 120, "flops": cells * 30 + cells // 8 * 10000}
    sf, sg = SIZES[c["storage"]]
    if kind == "monitor":
        return {"bytes": cells * (20 + 7 * sg), "flops": cells * 30}
    b = 2 * (c["q"] * sf + 7 * sg) * c["steps"]
    fl = FLOPS[c["q"]] * c["steps"]
    if kind == "closure":
        b += 28 + 8 * c["steps"] + 20
        fl += 10000
    if kind == "step":
        b += (20 if c["store"] else 0) + ((80 * c["steps"] + 28) if c["means"] else 0)
    return {"bytes": cells * b, "flops": cells * fl}


# ------------------------------------------------------------------ the same in 64 bits
_C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
      (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1), (1, 1, 1),
      (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)]


def _weight(q, n):
    order = sum(abs(v) for v in _C[q])
    return ((1 / 3, 1 / 18, 1 / 36) if n == 19 else (8 / 27, 2 / 27, 1 / 54, 1 / 216))[order]


def _at(a, c):
    """a at x + c, wrapped ([..., z, y, x])."""
    return torch.roll(a, (-c[2], -c[1], -c[0]), (-3, -2, -1)) if any(c) else a


def _feq(q, n, rho, u):
    w, c = _weight(q, n), _C[q]
    uu = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    cu = 3.0 * (c[0] * u[0] + c[1] * u[1] + c[2] * u[2])
    b = 1.0 - uu + cu + 0.5 * cu * cu
    if n == 27:
        b = b + cu * cu * cu / 6.0 - uu * cu
    return w * rho * b - w


def _fneq(q, n, p, u):
    """p: xx, yy, zz, xy, xz, yz."""
    w, c = _weight(q, n), _C[q]
    x, y, z = c
    h = ((x * x - 1 / 3) * p[0] + (y * y - 1 / 3) * p[1] + (z * z - 1 / 3) * p[2]
         + 2.0 * (x * y * p[3] + x * z * p[4] + y * z * p[5]))
    if n == 27:
        h = h + 3.0 * ((x * x * y - y / 3) * (p[0] * u[1] + 2 * u[0] * p[3]) + (x * x * z - z / 3) * (p[0] * u[2] + 2 * u[0] * p[4])
                       + (x * y * y - x / 3) * (p[1] * u[0] + 2 * u[1] * p[3]) + (y * y * z - z / 3) * (p[1] * u[2] + 2 * u[1] * p[5])
                       + (x * z * z - x / 3) * (p[2] * u[0] + 2 * u[2] * p[4]) + (y * z * z - y / 3) * (p[2] * u[1] + 2 * u[2] * p[5]))
        h = h + 6.0 * x * y * z * (u[0] * p[5] + u[1] * p[4] + u[2] * p[3])
    return 4.5 * w * h


def _noise(seed, step, cells):
    """The inlet's N(0, 1): Philox-4x32-10 at (cell, step, 0, 0) under the seed, Box-Muller."""
    m = np.uint64(0xFFFFFFFF)
    v = [np.asarray(cells, np.uint64), np.full(len(cells), step & 0xFFFFFFFF, np.uint64),
         np.full(len(cells), step >> 32, np.uint64), np.zeros(len(cells), np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        a, b = v[0] * np.uint64(0xD2511F53), v[2] * np.uint64(0xCD9E8D57)
        v = [(b >> np.uint64(32)) ^ v[1] ^ np.uint64(k0), b & m, (a >> np.uint64(32)) ^ v[3] ^ np.uint64(k1), a & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u1, u2 = (v[0].astype(np.float64) + 0.5) * 2.0 ** -32, v[1].astype(np.float64) * 2.0 ** -32
    return np.sqrt(-2.0 * np.log(u1)) * np.cos(2 * np.pi * u2)


class _Lattice:
    """The time step in 64 bits, population q of cell s holding what cell s + c_q reads next."""

    def __init__(self, v, fields):
        self.v = v
        self.n = v["q"]
        self.rho, ux, uy, uz, self.phi = (a.double().clone() for a in fields)
        self.u = [ux, uy, uz]
        nz, ny, nx = self.shape = tuple(self.rho.shape)
        self.p = [torch.zeros_like(self.rho) for _ in range(6)]
        fluid = torch.ones(self.shape, dtype=torch.bool, device=self.rho.device)
        if v["bc"] == "cross":
            fluid[:, :, (0, -1)] = False
            fluid[:, (0, -1), :] = False
        if v["bc"] != "box":
            fluid[(0, -1), :, :] = False
        self.fluid = fluid
        self.f, self.g = [], []
        for q in range(self.n):
            rho, u, _ = self._target(q)
            self.f.append(_feq(q, self.n, rho, u))
        for q in range(7):
            _, u, phi = self._target(q)
            cu = sum(c * a for c, a in zip(_C[q], u))
            self.g.append((0.25 if q == 0 else 0.125) * phi * (1.0 + 4.0 * cu))
        self.steps = 0
        self.nut = self.cs = None

    def _target(self, q):
        """rho, u, phi of x + c_q, of x itself where that leaves the lattice."""
        c, bc = _C[q], self.v["bc"]
        out = torch.zeros(self.shape, dtype=torch.bool, device=self.rho.device)
        for axis, d, open_ in ((2, c[0], bc == "cross"), (1, c[1], bc == "cross"), (0, c[2], bc != "box")):
            if d and open_:
                out.select(axis, self.shape[axis] - 1 if d > 0 else 0).fill_(True)
        pick = lambda a: torch.where(out, a, _at(a, c))  # noqa: E731
        return pick(self.rho), [pick(a) for a in self.u], pick(self.phi)

    def _grad(self, a):
        g = [torch.zeros_like(a) for _ in range(3)]
        for q in range(1, self.n):
            b = _at(a, _C[q])
            for d in range(3):
                if _C[q][d]:
                    g[d] += (3.0 * _weight(q, self.n) * _C[q][d]) * b
        return g

    @staticmethod
    def _unit(g):
        size = (g[0] * g[0] + g[1] * g[1] + g[2] * g[2]).sqrt()
        return [a / (size + 1e-9) for a in g], size

    def step(self):
        v, n = self.v, self.n
        phi = sum(_at(self.g[q], tuple(-a for a in _C[q])) for q in range(7))
        phi = torch.where(self.fluid, phi, torch.zeros_like(phi))
        nrm, size = self._unit(self._grad(phi))
        div = torch.zeros_like(phi)
        for q in range(1, n):
            for d in range(3):
                if _C[q][d]:
                    div += (3.0 * _weight(q, n) * _C[q][d]) * _at(nrm[d], _C[q])
        sigma = v["sigma"] if self.cs is None else v["sigma"] * self.cs
        F = [-sigma * div * size * a for a in nrm]
        seen, _ = self._unit(self._grad(torch.where(self.fluid, phi, self.phi)))
        s = torch.zeros_like(phi)
        j, t = [torch.zeros_like(phi) for _ in range(3)], [torch.zeros_like(phi) for _ in range(6)]
        pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
        for q in range(n):
            c = _C[q]
            a = _at(self.f[q], tuple(-b for b in c))
            s += a
            for d in range(3):
                if c[d]:
                    j[d] += c[d] * a
            for k, (d, e) in enumerate(pairs):
                if c[d] * c[e]:
                    t[k] += (c[d] * c[e]) * a
        rho = s + 1.0
        u = [(j[d] + 0.5 * F[d]) / rho for d in range(3)]
        p = [t[k] - rho * u[d] * u[e] + 0.5 * (u[d] * F[e] + u[e] * F[d]) for k, (d, e) in enumerate(pairs)]
        tr = (p[0] + p[1] + p[2]) / 3.0
        p = [p[0] - tr, p[1] - tr, p[2] - tr] + p[3:]
        nu = v["nu_water"] + phi * (v["nu_oil"] - v["nu_water"])
        if self.nut is not None:
            nu = nu + self.nut
        omco = 1.0 - 1.0 / (0.5 + 3.0 * nu)
        uF = u[0] * F[0] + u[1] * F[1] + u[2] * F[2]
        for q in range(n):
            c = _C[q]
            cF = sum(a * b for a, b in zip(c, F) if a)
            cu = sum(a * b for a, b in zip(c, u) if a)
            new = _feq(q, n, rho, u) + omco * _fneq(q, n, p, u) + _weight(q, n) * (1.5 * cF - 1.5 * uF + 4.5 * cu * cF)
            self.f[q] = torch.where(self.fluid, new, self.f[q])
        sharp = v["gamma"] * phi * (1.0 - phi)
        old = [_at(self.g[q], tuple(-a for a in _C[q])) for q in range(7)]
        for q in range(7):
            eq = 0.25 * phi if q == 0 else 0.125 * (phi + sum(c * (4.0 * phi * u[d] + sharp * seen[d]) for d, c in enumerate(_C[q]) if c))
            self.g[q] = torch.where(self.fluid, old[q] + v["omega_g"] * (eq - old[q]), self.g[q])
        for a, b in [(self.rho, rho), (self.phi, phi)] + list(zip(self.u, u)) + list(zip(self.p, p)):
            a.copy_(torch.where(self.fluid, b, a))
        if v["bc"] != "box":
            self._faces()
        self.steps += 1

    def _faces(self):
        v, n = self.v, self.n
        nz, ny, nx = self.shape
        cross = v["bc"] == "cross"
        dev = self.rho.device
        z, y, x = (torch.arange(k, device=dev) for k in (nz, ny, nx))
    
        def write(axis, at, q, where, rho, u, omco, inner):
            """f_eq(rho, u) + omco f_neq of the inner plane's neighbour into population q of a face."""
            pl = lambda a: a.select(axis, inner)  # noqa: E731
            c = [_C[q][2], _C[q][1], _C[q][0]]
            del c[axis]
            sh = lambda a: torch.roll(pl(a), (-c[0], -c[1]), (0, 1))  # noqa: E731
            val = _feq(q, n, rho, u) + omco * _fneq(q, n, [sh(a) for a in self.p], [sh(a) for a in self.u])
            face = self.f[q].select(axis, at)
            face.copy_(torch.where(where, val, face))

        def inside(q, axis, fluid_only):
            """Face cells whose neighbour along c_q stays in the lattice (in its fluid range)."""
            dims = [d for d in range(3) if d != axis]
            ok = None
            for i, d in enumerate(dims):
                k = self.shape[d]
                r = torch.arange(k, device=dev) + (_C[q][2], _C[q][1], _C[q][0])[d]
                open_ = d == 0 or cross  # z, and with the crossflow x and y
                m = torch.ones(k, dtype=torch.bool, device=dev)
                if open_:
                    m = (r >= (1 if fluid_only else 0)) & (r <= (k - 2 if fluid_only else k - 1))
                m = m[:, None] if i == 0 else m[None, :]
                ok = m if ok is None else ok & m
            return ok

        one = torch.ones((), dtype=torch.float64, device=dev)
        if cross:
            disc = (z[:, None] - v["water_cz"]) ** 2 + (x[None, :] - v["water_cx"]) ** 2 <= v["water_r2"]
            for a, b in ((self.rho, 1.0), (self.phi, 0.0), (self.u[0], 0.0), (self.u[1], v["u_water"]), (self.u[2], 0.0)):
                a[:, 0, :] = torch.where(disc, b * one, a[:, 0, :])
            for q in range(n):
                if _C[q][1] == 1:
                    write(1, 0, q, disc & inside(q, 1, False), one, [0 * one, v["u_water"] * one, 0 * one], v["omco"], 1)
            self.g[3][:, 0, :] = torch.where(disc, 0 * one, self.g[3][:, 0, :])
        disc = (y[:, None] - v["oil_cy"]) ** 2 + (x[None, :] - v["oil_cx"]) ** 2 <= v["oil_r2"]
        speed = torch.full((ny, nx), v["u_oil"], dtype=torch.float64, device=dev)
        if v["noise"]:
            cells = disc.reshape(-1).nonzero().reshape(-1)
            k = torch.as_tensor(_noise(v["seed"], self.steps, cells.cpu().numpy()), device=dev)
            speed.view(-1)[cells] = v["u_oil"] * (1.0 + v["noise"] * k)
        for a, b in ((self.rho, one), (self.phi, one), (self.u[0], 0 * one), (self.u[1], 0 * one), (self.u[2], speed)):
            a[0] = torch.where(disc, b, a[0])
        for q in range(n):
            if _C[q][2] == 1:
                write(0, 0, q, disc & inside(q, 0, True), one, [0 * one, 0 * one, speed], v["omco_oil"], 1)
        self.g[5][0] = torch.where(disc, 0.125 * (1.0 + 4.0 * speed), self.g[5][0])
        for axis, sign_q in ((1, 4), (0, 6)):
            if axis == 1 and not cross:
                continue
            k = self.shape[axis]
            mask = self.fluid.select(axis, k - 2)
            for a in (self.rho, self.phi, *self.u):
                a.select(axis, k - 1).copy_(torch.where(mask, a.select(axis, k - 2), a.select(axis, k - 1)))
            rho, phi = self.rho.select(axis, k - 1), self.phi.select(axis, k - 1)
            u = [a.select(axis, k - 1) for a in self.u]
            for q in range(n):
                if (_C[q][1] if axis == 1 else _C[q][2]) == -1:
                    write(axis, k - 1, q, mask & inside(q, axis, axis == 1), rho, u, v["omco"], k - 2)
            face = self.g[sign_q].select(axis, k - 1)
            face.copy_(torch.where(mask, 0.125 * phi * (1.0 - 4.0 * (u[1] if axis == 1 else u[2])), face))
        if cross:  # periodic x by copies
            for q in range(n):
                c = _C[q]
                if not c[0]:
                    continue
                ok = torch.zeros((nz, ny), dtype=torch.bool, device=dev)
                ok[max(0, -c[2]):nz - max(0, c[2]), max(0, -c[1]):ny - max(0, c[1])] = True
                to, src = (0, nx - 3) if c[0] > 0 else (nx - 1, 2)
                self.f[q][:, :, to] = torch.where(ok, self.f[q][:, :, src], self.f[q][:, :, to])
            self.g[1][:, :, 0] = self.g[1][:, :, nx - 3]
            self.g[2][:, :, nx - 1] = self.g[2][:, :, 2]
            for a in (self.phi, *self.u):
                a[:, :, 0], a[:, :, nx - 1] = a[:, :, nx - 2].clone(), a[:, :, 1].clone()

    def out(self):
        return {"f": torch.stack(self.f).reshape(-1), "g": torch.stack(self.g).reshape(-1)}

    def macros(self):
        return {"rho": self.rho.reshape(-1), "ux": self.u[0].reshape(-1), "uy": self.u[1].reshape(-1),
                "uz": self.u[2].reshape(-1), "phi": self.phi.reshape(-1)}


def _f32(x):
    return float(np.float32(x))


def _values(c, seed):
    """The step's parameters as plain numbers, rounded to the 32 bits that the call takes them in."""
    bc = c.get("bc", "jet")
    if bc == "cross":
        d = max(6, min(c["nx"], c["ny"]) // 8)
        u, r2 = _f32(0.05), float((d // 2) ** 2)
        nw, no = _f32(u * d / (3.0 * d)), _f32(u * d / (2.5 * d))
        return {"bc": bc, "q": c["q"], "nu_water": nw, "nu_oil": no, "omco": 1 - 1 / (0.5 + 3 * nw), "omco_oil": 1 - 1 / (0.5 + 3 * no),
                "sigma": _f32(u * u * d / (2.5 * d)), "gamma": 0.5, "omega_g": 1.0, "u_oil": u, "u_water": u, "noise": 0.0, "seed": 0,
                "oil_cx": (c["nx"] - 1) * 0.5, "oil_cy": _f32((c["ny"] - 1) * 0.25), "oil_r2": r2,
                "water_cx": (c["nx"] - 1) * 0.5, "water_cz": _f32(np.float32(0.7) * np.float32((c["nz"] - 1) * 0.5)), "water_r2": r2}
    return _jet_numbers(bc, c["nx"], c["ny"], c.get("q", 19), _jet_values(c), seed)


def _jet_numbers(bc, nx, ny, q, v, seed):
    nu = _f32((v["tau"] - 0.5) / 3.0)
    om = 1 - 1 / (0.5 + 3 * nu)
    return {"bc": bc, "q": q, "nu_water": nu, "nu_oil": nu, "omco": om, "omco_oil": om, "sigma": _f32(v["sigma"]),
            "gamma": _f32(4.0 * v["mobility"] / (v["width"] * 0.25)), "omega_g": _f32(1.0 / (0.5 + v["mobility"] / 0.25)),
            "u_oil": _f32(v["w_in"]), "noise": _f32(v["noise"]), "seed": seed, "oil_cx": (nx - 1) * 0.5, "oil_cy": (ny - 1) * 0.5,
            "oil_r2": float((v["diam"] // 2) ** 2)}


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))


def _split(net):
    """W1, b1, W2, b2, W3, b3, mean, 1/std, scale, offset of a network buffer."""
    out, o = [], 0
    for shape in ((64, 16), (64,), (64, 64), (64,), (2, 64), (2,), (12,), (12,), (2,), (2,)):
        k = math.prod(shape)
        out.append(net[o:o + k].reshape(shape))
        o += k
    return out


def _predict(net, feats):
    w1, b1, w2, b2, w3, b3, mean, inv, scale, offset = _split(net)
    got = []
    for x in feats.split(1 << 20):
        h = _gelu(((x - mean) * inv) @ w1[:, :12].T + b1)
        got.append((_gelu(h @ w2.T + b2) @ w3.T + b3) * scale + offset)
    return torch.cat(got)


def _diff(a, axis, per):
    """Central difference along an axis of [z][y][x]: wrapped, or clamped at the faces."""
    up, dn = torch.roll(a, -1, axis), torch.roll(a, 1, axis)
    if not per:
        k = a.shape[axis]
        up.select(axis, k - 1).copy_(a.select(axis, k - 1))
        dn.select(axis, 0).copy_(a.select(axis, 0))
    return 0.5 * (up - dn), up + dn


def _features(rho, u, phi, nu):
    """The twelve inputs of the closure network on an x, y periodic jet."""
    per = (False, True, True)  # z, y, x
    d = [[_diff(a, 2 - k, per[2 - k])[0] for k in range(3)] for a in u]
    g = [_diff(phi, 2 - k, per[2 - k]) for k in range(3)]
    lap = sum(b for _, b in g) - 6.0 * phi
    size = sum(a * a for a, _ in g).sqrt()
    nrm = [a / (size + 1e-9) for a, _ in g]
    S = [[0.5 * (d[a][b] + d[b][a]) for b in range(3)] for a in range(3)]
    ss = sum(S[a][b] ** 2 for a in range(3) for b in range(3))
    nsn = sum(nrm[a] * S[a][b] * nrm[b] for a in range(3) for b in range(3))
    w = (d[2][1] - d[1][2]) ** 2 + (d[0][2] - d[2][0]) ** 2 + (d[1][0] - d[0][1]) ** 2
    f = torch.stack([phi, 4 * phi * (1 - phi), size, lap, (2 * ss).sqrt(), w.sqrt(), nsn, (u[0] ** 2 + u[1] ** 2 + u[2] ** 2).sqrt(),
                     u[2], rho - 1, d[0][0] + d[1][1] + d[2][2], torch.full_like(phi, nu)], -1)
    return f.reshape(-1, 12), S, size


def _exact_train(c, seed):
    net = torch.as_tensor(_net_values(seed), device="cuda").double()
    P = 5378
    feats, targets, weights = _rows(c, seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    b = min(c["batch"], c["rows"])
    m, v, avg = torch.zeros(P, device="cuda").double(), torch.zeros(P, device="cuda").double(), net[:P].clone()
    for t in range(1, c["steps"] + 1):
        i = torch.randint(0, c["rows"], (b,), device="cuda", generator=g)
        p = net[:P].clone().requires_grad_()
        w1, b1, w2, b2, w3, b3, mean, inv, scale, offset = _split(torch.cat((p, net[P:])))
        h = _gelu(((feats[i].double() - mean) * inv) @ w1[:, :12].T + b1)
        r = _gelu(h @ w2.T + b2) @ w3.T + b3
        loss = (weights[i].double() * (r - (targets[i].double() - offset) / scale) ** 2).sum() / b
        grad, = torch.autograd.grad(loss, p)
        m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
        net[:P] -= 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
        avg = 0.9999 * avg + 0.0001 * net[:P]
    net[:P] = avg
    return {"net": net, "grad": grad, "m": m, "v": v, "loss": loss.detach().reshape(1)}


def _exact_data(c, seed):
    rho, ux, uy, uz, phi = (a.double() for a in _fields((c["nz"], c["ny"], c["nx"]), seed, "jet", 0.05, _diam(c)))
    v = _values(c, seed)

    def mean(a):
        nz, ny, nx = a.shape
        return a.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2).mean((1, 3, 5))

    u = [ux, uy, uz]
    g = [_diff(phi, axis, per)[0] for axis, per in ((2, True), (1, True), (0, False))]
    area = mean(sum(a * a for a in g).sqrt())
    cr, cu, cp = mean(rho), [mean(a) for a in u], mean(phi)
    pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
    tau = [mean(u[a] * u[b]) - cu[a] * cu[b] for a, b in pairs]
    feats, S, size = _features(cr, cu, cp, _f32(_f32(v["nu_water"]) * 0.5))
    tr = (tau[0] + tau[1] + tau[2]) / 3
    t = {p: tau[k] - (tr if p[0] == p[1] else 0) for k, p in enumerate(pairs)}
    num = sum(t[(min(a, b), max(a, b))] * S[a][b] for a in range(3) for b in range(3))
    den = sum(S[a][b] ** 2 for a in range(3) for b in range(3))
    nut = (-num / (2 * den + 1e-12)).clamp(-NUT_MAX, NUT_MAX)
    cs = torch.where(size >= 1e-2, (2 * area / size.clamp_min(1e-30)).clamp(0.25, 4.0), torch.ones_like(size))
    net = torch.as_tensor(_net_values(seed), device="cuda").double()
    return {"coarse": torch.stack([cr, *cu, cp]).reshape(-1), "tau": torch.stack(tau).reshape(-1), "area": area.reshape(-1),
            "targets": torch.stack([nut, cs], -1).reshape(-1, 2),
            "weights": torch.stack([torch.ones_like(cp), 4 * cp * (1 - cp) + 0.01], -1).reshape(-1, 2),
            "feats": feats, "predicted": _predict(net, feats)}


def _exact_monitor(c, seed):
    shape = nz, ny, nx = c["nz"], c["ny"], c["nx"]
    fields = _fields(shape, seed, "jet", 0.05, _diam(c))
    lat = _Lattice(_values(c, seed), fields)
    fl = lat.fluid
    kind = {"f32": torch.float32, "f16g32": torch.float32, "f16": torch.float16, "bf16": torch.float16}[c["storage"]]
    g = [a.float().to(kind).double() for a in lat.g]
    nxt = sum(_at(g[q], tuple(-a for a in _C[q])) for q in range(7))[fl].sum()
    rho, phi, u = lat.rho[fl], lat.phi[fl], [a[fl] for a in lat.u]
    u2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    sums = [phi.sum(), nxt, rho.sum(), *((rho * a).sum() for a in u), (0.5 * rho * u2).sum(), u2.max().sqrt(), 0.0, float(fl.sum())]
    flux = [g[5][0].sum() + g[6][-1].sum(), g[6][1].sum() + g[5][-2].sum()]
    axis = lambda a: a[:, (ny - 1) // 2:ny // 2 + 1, (nx - 1) // 2:nx // 2 + 1].mean((1, 2))  # noqa: E731
    on = fl & (lat.phi > 0.5)
    none = nz * ny * nx
    label = torch.where(on, torch.arange(none, device=on.device).reshape(shape), none)
    while True:  # the smallest index of the component spreads over its cells
        new = label
        for c3 in _C[1:7]:
            s = _at(label, c3)
            new = torch.minimum(new, torch.where(on, s, new))
        new = torch.where(on, torch.minimum(new, torch.cat((new.reshape(-1), new.new_full((1,), none)))[new.clamp_max(none)]), new)
        if torch.equal(new, label):
            break
        label = new
    root, inv, cells = torch.unique(label[on], return_inverse=True, return_counts=True)
    volume = torch.zeros(len(root), dtype=torch.float64, device=on.device).index_add_(0, inv, lat.phi[on])
    first = torch.zeros(len(root), dtype=torch.int64, device=on.device)
    first[torch.unique(torch.searchsorted(root, label[1][on[1]]))] = 1
    return {"sums": torch.tensor([float(a) for a in sums], dtype=torch.float64), "flux": torch.stack(flux), "uz": axis(lat.u[2]),
            "phi": axis(lat.phi)} | {k: torch.as_tensor(_padded(a.cpu().numpy())) for k, a in
                                     (("root", root), ("cells", cells), ("volume", volume), ("inlet", first))}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "train":
        return _exact_train(c, seed)
    if kind == "data":
        return _exact_data(c, seed)
    if kind == "monitor":
        return _exact_monitor(c, seed)
    if kind == "sweep":
        rng, out, cells = np.random.default_rng(c["set"]), [], 0
        for i in range(c["count"]):  # the draws of sweep_params
            k = int(rng.choice([32, 48, 64, 96]))
            v = {"w_in": float(rng.uniform(0.02, 0.08)), "diam": int(rng.integers(6, 13)), "sigma": float(10 ** rng.uniform(-4, -2)),
                 "tau": float(rng.uniform(0.51, 0.6)), "mobility": float(rng.uniform(0.05, 0.2)), "width": 4.0, "noise": 0.01}
            cells += 4 * k ** 3
            r = v["diam"] // 2
            lat = _Lattice(_jet_numbers("jet", k, k, c["q"], v, 1000 * c["set"] + i),
                           _fields((4 * k, k, k), 1000 * seed + i, "jet", _f32(v["w_in"]), max(2 * r, 4)))
            for _ in range(c["steps"]):
                lat.step()
            out.append(lat.out())
        return out
    if c["nx"] * c["ny"] * c["nz"] > 20_000_000:
        return None  # more memory and time than a check should take
    lat = _Lattice(_values(c, seed), _fields((c["nz"], c["ny"], c["nx"]), seed, c.get("bc", "jet"), 0.05, _diam(c)))
    if kind == "closure":
        nu = lat.v["nu_water"]
        out = _predict(torch.as_tensor(_net_values(seed), device="cuda").double(), _features(lat.rho, lat.u, lat.phi, nu)[0])
        lat.nut = out[:, 0].clamp(max(-0.5 * nu, -NUT_MAX), NUT_MAX).reshape(lat.shape)
        lat.cs = out[:, 1].clamp(0.25, 4.0).reshape(lat.shape)
        for _ in range(c["steps"]):
            lat.step()
        return lat.out() | lat.macros() | {"nut": lat.nut.reshape(-1), "cs": lat.cs.reshape(-1)}
    means = {}
    for t in range(1, c["steps"] + 1):
        lat.step()
        if c["means"]:
            u = [a.reshape(-1) for a in lat.u]
            now = {"avg_phi": lat.phi.reshape(-1), "avg_ux": u[0], "avg_uy": u[1], "avg_uz": u[2], "avg_uxux": u[0] * u[0],
                   "avg_uyuy": u[1] * u[1], "avg_uzuz": u[2] * u[2], "avg_uxuy": u[0] * u[1], "avg_uxuz": u[0] * u[2],
                   "avg_uyuz": u[1] * u[2]}
            means = {k: means.get(k, 0.0) + (a - means.get(k, 0.0)) / t for k, a in now.items()}
    out = lat.out()
    if c["store"]:
        out |= lat.macros()
    if c["means"]:
        d = [[0.5 * (torch.roll(a, -1, 2 - k) - torch.roll(a, 1, 2 - k)) for k in range(3)] for a in lat.u]
        inner = torch.zeros(lat.shape, dtype=torch.bool, device=lat.rho.device)
        inner[1:-1, 1:-1, 1:-1] = True
        w = [torch.where(inner, a, torch.zeros_like(a)) for a in (d[2][1] - d[1][2], d[0][2] - d[2][0], d[1][0] - d[0][1])]
        means |= {"vort_x": w[0].reshape(-1), "vort_y": w[1].reshape(-1), "vort_z": w[2].reshape(-1),
                  "vort_mag": (w[0] ** 2 + w[1] ** 2 + w[2] ** 2).sqrt().reshape(-1)}
        out |= means
    return out
