"""Workloads that the framework's speed is judged by, from the smallest calls
to the eight-block case that bench.py runs by default.

A case is a dict of plain values.  Kinds:

  cycles    GpuSolver.cycles on one bump-channel block: whole iterations
            (residual, implicit stage, update, boundary), with or without
            multigrid levels, laminar or k-omega SST, LU-SGS or DDADI, FP64
            or the FP32 implicit stage
  blocks    GpuSolver.cycles_all on the bump channel cut into eight uneven
            1:1-patched blocks with multigrid levels
  box       GpuSolver.cycles_all on a periodic box of blocks, inviscid
  stages    the iteration driven stage by stage, as a host program that
            keeps its own iteration loop calls it
  residual  the residual stage alone (RESIDI of a host program)
  train     one training step of the learned warm start
  setup     metrics and wall distance of a block and its levels from nodes

Every state comes from the seed: a free stream with a boundary layer of a
seeded thickness and seeded density noise, as a run meets it after its first
iterations.
"""
import math

import numpy as np
import torch

from finflo_b200 import case as ffcase
from finflo_b200 import grid, warmstart
from finflo_b200.gpu import GpuSolver
from finflo_b200.case import SLOT, FFParams


def listed():
    return [
        # the smallest block anybody runs: latency and launches only
        _cycles("laminar_16x8x8", 16, 8, 8, cycles=10),
        # the laminar bump of the tests and of the warm-start family
        _cycles("laminar_64x32x32", 64, 32, 32, cycles=5),
        # the reference's default implicit stage, odd sizes
        _cycles("laminar_ddadi_57x35x21", 57, 35, 21, ddadi=True, cycles=5),
        # the k-omega SST V-cycle that the convergence studies run
        _cycles("sst_vcycle_128x64x64", 128, 64, 64, levels=3, sst=True, inter=1, cycles=2),
        # the same method with the FP32 implicit stage and FP32 coarse levels, a ragged block
        _cycles("sst_vcycle_fp32_104x56x40", 104, 56, 40, levels=3, sst=True, inter=1, fp32=True, cycles=2),
        # DDADI with k-omega on a single grid
        _cycles("sst_ddadi_90x50x34", 90, 50, 34, sst=True, ddadi=True, inter=1, cycles=3),
        # a host program that calls the stages itself
        {"name": "sst_stages_72x40x24", "kind": "stages", "ni": 72, "nj": 40, "nk": 24, "sst": True, "inter": 1},
        # the residual stage as a drop-in
        {"name": "sst_residual_128x64x64", "kind": "residual", "ni": 128, "nj": 64, "nk": 64, "sst": True, "inter": 1},
        # many blocks of uneven size, FP32 implicit stage, no viscosity
        {"name": "box_3x2x2_fp32", "kind": "box", "bi": 3, "bj": 2, "bk": 2, "cells": 1200000, "layout": 2, "fp32": True,
         "cycles": 1},
        # the largest: the eight-block SST bump, 16.8M cells, plain FP64
        {"name": "sst_blocks_512x256x128", "kind": "blocks", "ni": 512, "nj": 256, "nk": 128, "levels": 3, "layout": 5,
         "fp32": False, "cycles": 1},
        # training of the learned warm start at its batch size
        {"name": "warm_start_step_16", "kind": "train", "batch": 16},
        # a new geometry: metrics of three levels and the wall distance
        {"name": "setup_128x64x64", "kind": "setup", "ni": 128, "nj": 64, "nk": 64, "levels": 3},
    ]


def _cycles(name, ni, nj, nk, levels=1, sst=False, ddadi=False, fp32=False, inter=3, cycles=1):
    return {"name": name, "kind": "cycles", "ni": ni, "nj": nj, "nk": nk, "levels": levels, "sst": sst, "ddadi": ddadi,
            "fp32": fp32, "inter": inter, "cycles": cycles}


def _size(rng, lo, hi, step=1):
    """A size between lo and hi, even over its logarithm, a multiple of step."""
    return max(step, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    kind = rng.choice(["cycles", "cycles", "cycles", "stages", "residual", "box", "blocks", "train", "setup"])
    if kind == "cycles":
        levels = rng.choice([1, 1, 2, 3])
        q = 2 ** (levels - 1)
        lo = 16 if levels == 3 else 8
        sst = rng.random() < 0.6
        c = _cycles("", _size(rng, max(lo, 12), 160, q), _size(rng, lo, 96, q), _size(rng, lo, 80, q), levels, sst,
                    rng.random() < 0.3, rng.random() < 0.35, rng.choice([1, 3]) if not sst else 1, rng.randint(1, 6))
        del c["name"]
        return c
    if kind in ("stages", "residual"):
        return {"kind": kind, "ni": _size(rng, 12, 160), "nj": _size(rng, 8, 96), "nk": _size(rng, 6, 80),
                "sst": rng.random() < 0.7, "inter": rng.choice([1, 3])}
    if kind == "box":
        return {"kind": "box", "bi": rng.randint(2, 4), "bj": rng.randint(1, 3), "bk": 2,
                "cells": _size(rng, 150000, 1500000), "layout": rng.randint(1, 50), "fp32": rng.random() < 0.6,
                "cycles": rng.randint(1, 3)}
    if kind == "blocks":
        return {"kind": "blocks", "ni": _size(rng, 64, 256, 8), "nj": _size(rng, 48, 128, 8), "nk": _size(rng, 32, 96, 8),
                "levels": rng.choice([2, 3]), "layout": rng.randint(1, 50), "fp32": rng.random() < 0.5,
                "cycles": rng.randint(1, 3)}
    if kind == "train":
        return {"kind": "train", "batch": rng.randint(2, 24)}
    return {"kind": "setup", "ni": _size(rng, 24, 160, 4), "nj": _size(rng, 16, 96, 4), "nk": _size(rng, 12, 80, 4),
            "levels": 3}


# ---- inputs -----------------------------------------------------------------

STATE = ("TEMP", "U", "V", "W", "PDIFF", "EPS2", "VIST")
TURB = ("RK", "REPS", "RKOLD", "EPSOLD")
RESID = ("DRO", "DM", "DN", "DW", "DE")


def _developed(blk, fs, rng, sst):
    """A boundary layer of seeded thickness on both walls (y in the index
    space of the stretched grid) and smooth pressure and cross-flow waves."""
    kmax, jmax, imax = blk.kmax, blk.jmax, blk.imax
    delta = rng.uniform(0.08, 0.2)
    ph = rng.uniform(0.0, 2.0 * np.pi, 3)
    j = (np.arange(jmax) + 0.5) / jmax
    d = np.minimum(j, 1.0 - j) if not sst else j
    prof = np.tanh(d / delta)[None, :, None]
    x = (np.arange(imax) + 0.5)[None, None, :] / imax
    z = (np.arange(kmax) + 0.5)[:, None, None] / kmax
    wave = np.sin(2 * np.pi * x + ph[0]) * np.cos(np.pi * z + ph[1])
    one = np.ones((kmax, jmax, imax))
    blk.interior("U")[:] = fs["u"] * prof * (1.0 + 0.01 * wave)
    blk.interior("V")[:] = 0.01 * fs["u"] * prof * np.sin(2 * np.pi * x + ph[2]) * one
    blk.interior("W")[:] = 0.005 * fs["u"] * prof * wave
    blk.interior("PDIFF")[:] = 0.01 * fs["p"] * np.cos(2 * np.pi * x + ph[0]) * one
    if sst:
        rk, re = ffcase.sst_freestream(fs)
        hump = (np.exp(-((d - 0.5 * delta) / (0.4 * delta)) ** 2))[None, :, None]
        blk.interior("RK")[:] = rk * (1.0 + 50.0 * hump) * (1.0 + 0.05 * wave)
        blk.interior("REPS")[:] = re * (1.0 + 100.0 * np.exp(-d / (0.3 * delta))[None, :, None]) * one
        blk.arrays["RKOLD"][:] = blk.arrays["RK"]
        blk.arrays["EPSOLD"][:] = blk.arrays["REPS"]


def _channel(c, seed):
    """(levels, parameters per level, nodes, wall points) of a bump channel
    whose metrics and wall distance the device fills."""
    sst, nlev = c.get("sst", False), c.get("levels", 1)
    rng = np.random.default_rng(seed)
    fc = ffcase.FlowConditions(mach=0.6, reynolds=1e6) if sst else ffcase.FlowConditions(mach=0.5, reynolds=1e4)
    fs = fc.freestream()
    X, Y, Z = grid.bump_nodes(c["ni"] + 1, c["nj"] + 1, c["nk"] + 1, h1=2e-6 if sst else min(1e-3, 0.3 / c["nj"]), amp=0.1)
    levels = []
    for lv in range(nlev):
        m = grid.Metrics(c["ni"] >> lv, c["nj"] >> lv, c["nk"] >> lv)
        m.arrays = {n: np.zeros(m.ntot) for n in grid.METRIC_NAMES}
        blk = ffcase.block_from_metrics(m, ffcase.channel_patches(m.imax, m.jmax, m.kmax, fs))
        ffcase.init_freestream(blk, fs, noise=1e-3 if lv == 0 else 0.0, seed=seed)
        levels.append(blk)
    prm = ffcase.make_params(fc, levels[0].dims, cfl=1.0 if sst else 2.0, cfll=1.0 if sst else 2.0, inter=c.get("inter", 3))
    if sst:
        for lv, blk in enumerate(levels):
            ffcase.setup_sst(blk, prm if lv == 0 else FFParams.from_buffer_copy(prm), fs, distw=False)
    _developed(levels[0], fs, rng, sst)
    prms = [ffcase.level_params(prm, lv + 1) for lv in range(nlev)]
    for lv, q in enumerate(prms):
        q.predgs_full = 1
        q.ddadi = int(c.get("ddadi", False))
        q.lusgs_fp32 = int(c.get("fp32", False))
        q.res_fp32 = int(c.get("fp32", False) and lv > 0)
    return levels, prms, (X, Y, Z), ffcase.wall_points((X, Y, Z), levels[0].patches)


def _solver(c, seed):
    levels, prms, nodes, walls = _channel(c, seed)
    g = GpuSolver(0)
    bid = g.add_levels(levels, prms) if len(levels) > 1 else g.add_block(levels[0], prms[0])
    for q, blk in enumerate(levels):
        g.upload(bid + q, STATE + (TURB if c.get("sst") else ()))
        blk.arrays = {}
    g.block_metrics_levels(bid, len(levels), *nodes)
    if c.get("sst"):
        g.wall_distance(bid, walls)
    g.start(bid)
    return {"g": g, "bid": bid, "case": c}


def _box_sizes(c):
    nb = (c["bi"], c["bj"], c["bk"])
    return ffcase.box_block_sizes(nb, seed=c["layout"], target=c["cells"], tol=0.35,
                                  nodes=tuple(range(17, 98, 4)) if c["cells"] > 6e5 else tuple(range(13, 62, 4)))


def prepare(c, seed):
    kind = c["kind"]
    if kind in ("cycles", "stages", "residual"):
        return _solver(c, seed)
    if kind == "box":
        blocks, prms, fs = ffcase.periodic_box_case(sizes=_box_sizes(c), nb=(c["bi"], c["bj"], c["bk"]), seed=seed,
                                                    lusgs_fp32=c["fp32"])
        g = GpuSolver(0)
        ids = g.add_multiblock([[b] for b in blocks], [[p] for p in prms])
        ph = np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, 3)
        for bid, b in zip(ids, blocks):
            x, y, z = (2.0 * np.pi * b.interior(n) for n in ("XC", "YC", "ZC"))
            b.interior("PDIFF")[:] = 0.01 * fs["p"] * np.sin(x + ph[0]) * np.cos(y)
            b.interior("U")[:] *= 1.0 + 0.05 * np.sin(y + ph[1])
            b.interior("W")[:] *= 1.0 + 0.05 * np.cos(z + ph[2]) * np.sin(x)
            g.upload(bid, STATE + tuple(grid.METRIC_NAMES))
            b.arrays = {}
        g.start_all()
        return {"g": g, "ids": ids, "case": c}
    if kind == "blocks":
        it = ffcase.bump_multiblock_blocks(cells=(c["ni"], c["nj"], c["nk"]), nb=(2, 2, 2), nlev=c["levels"],
                                           seed=c["layout"], inter=1, lusgs_fp32=c["fp32"], coarse_fp32=c["fp32"],
                                           coarse_res_fp32=c["fp32"], noise=0.0, device_setup=True)
        _, fs = next(it)
        walls = next(it)[1]
        g = GpuSolver(0)
        rng = np.random.default_rng(seed)
        ids = []
        for n, (levels, prms) in enumerate(it):
            for q in prms:
                q.predgs_full = 1
            for pa in levels[0].patches:   # this context's ids: the levels of a block follow one another
                if pa.ityp == grid.BC_CON:
                    pa.ibtype *= c["levels"]
            noise = rng.standard_normal((levels[0].kmax, 1, levels[0].imax))
            levels[0].interior("TEMP")[:] = fs["t"] * (1.0 - 1e-3 * noise)
            wave = np.sin(np.arange(levels[0].jmax) * rng.uniform(0.02, 0.1) + rng.uniform(0.0, 6.0))
            levels[0].interior("V")[:] = 0.01 * fs["u"] * wave[None, :, None]
            ids.append(g.add_levels(levels, prms))
            for q, blk in enumerate(levels):
                g.upload(ids[-1] + q, STATE + TURB)
            g.block_metrics_levels(ids[-1], c["levels"], *levels[0].nodes)
            g.wall_distance(ids[-1], walls)
            for blk in levels:
                blk.arrays = {}
                blk.nodes = None
        g.start_all()
        return {"g": g, "ids": ids, "case": c}
    if kind == "train":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        net = warmstart.WarmStartNet(seed=seed % 1000003)
        x = torch.zeros(c["batch"], warmstart.IN_PAD, device="cuda")
        x[:, :2] = torch.rand(c["batch"], 2, generator=gen, device="cuda") * 2 - 1
        n = net.spec.ncell
        s = torch.linspace(0, 6.0, n, device="cuda")
        amp = torch.randn(c["batch"], 1, net.spec.nvar, generator=gen, device="cuda")
        t = amp * torch.sin(s)[None, :, None] + 0.1 * torch.randn(c["batch"], n, net.spec.nvar, generator=gen, device="cuda")
        return {"net": net, "x": x, "t": t.reshape(-1, net.spec.nvar).contiguous(), "case": c}
    levels, prms, (X, Y, Z), walls = _channel(c, seed)
    r = np.random.default_rng(seed)
    Y = Y * (1.0 + 0.01 * r.random()) + 1e-4 * np.sin(X * 3.0 + r.uniform(0, 6.0))   # another geometry for every seed
    g = GpuSolver(0)
    bid = g.add_levels(levels, prms)
    return {"g": g, "bid": bid, "nodes": (X, Y, Z), "walls": ffcase.wall_points((X, Y, Z), levels[0].patches), "case": c}


class _Slot:
    """A device array of the library for torch, without a copy."""

    def __init__(self, g, bid, name):
        self.keep = g
        self.__cuda_array_interface__ = {"data": (g.device_ptr(bid, name), False), "shape": (g.blocks[bid][0].ntot,),
                                         "typestr": "<f8", "version": 3}


def _slots(g, bid, names):
    return {n: torch.as_tensor(_Slot(g, bid, n), device="cuda") for n in names}


# ---- one pass ---------------------------------------------------------------

FIELDS = ("TEMP", "U", "V", "W", "PDIFF")


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "train":
        net = s["net"]
        net.forward(s["x"])
        loss = net.backward(s["t"])
        net.adam(2e-3)
        return {"pred": net.pred, "loss": loss, "grad": net.g, "w": net.w}
    g = s["g"]
    if kind in ("box", "blocks"):
        hist = g.cycles_all(c["cycles"], icycle0=2)
        names = FIELDS + (("RK", "REPS") if kind == "blocks" else ())
        fields = [_slots(g, b, names) for b in s["ids"]]
        if len(fields) * len(names) > 60:   # one array per variable over all blocks
            fields = {n: torch.cat([f[n] for f in fields]) for n in names}
        return {"hist": hist, "fields": fields}
    bid = s["bid"]
    names = FIELDS + (("RK", "REPS") if c.get("sst") else ())
    if kind == "cycles":
        return {"hist": g.cycles(c["cycles"], bid, icycle0=2), "fields": _slots(g, bid, names)}
    if kind == "stages":
        g.statim(bid)
        g.residu(bid, 1, 2)
        r = g.resl2(bid)
        g.imps(bid, 1)
        d = g.fin(bid)
        g.boundi(bid)
        return {"resl2": r, "dromax": d, "fields": _slots(g, bid, names)}
    if kind == "residual":
        g.residu(bid, 1, 2)
        return _slots(g, bid, RESID + (("DRK", "DEPS") if c["sst"] else ()))
    g.block_metrics_levels(bid, c["levels"], *s["nodes"])
    g.wall_distance(bid, s["walls"])
    return [_slots(g, bid + q, grid.METRIC_NAMES + ("DISTW",)) for q in range(c["levels"])]


# ---- the least work ---------------------------------------------------------

def work(c):
    """Bytes: every cell's state and metrics read once and its state written
    once a cycle (the residual stage: state and metrics in, residual out).
    Flops: a residual (three faces a cell), the implicit stage's sweeps and
    the update, per cell and cycle; a V-cycle evaluates the fine residual
    twice and adds 1/7 for the coarse levels."""
    kind = c["kind"]
    if kind == "train":
        _, nparam = warmstart.layers(warmstart.BUMP)
        rows, v, flops = c["batch"], 0.0, 0.0
        vox = rows * 16
        for l in warmstart.layers(warmstart.BUMP)[0]:
            if l.name.startswith("enc"):
                m = rows
            elif l.name.startswith("up"):
                m = vox
                vox *= 8
            else:
                m = vox
            flops += 6.0 * m * l.n * l.k
            v += m * l.n
        # activations written once forward and read once backward in 16 bits,
        # targets and prediction in 32, weights with both moments and gradient
        return {"bytes": 2 * 2 * v + 4 * vox * (5 + 16) + 4.0 * nparam * 8, "flops": flops}
    n = float(c["cells"]) if kind == "box" else float(c["ni"] * c["nj"] * c["nk"])
    sst = c.get("sst", kind == "blocks")
    nv = 7 if sst else 5
    if kind == "setup":
        pts = 2.0 * c["ni"] * c["nk"]
        return {"bytes": n * 8 * (3 + 20) * 8 / 7 + 24 * pts, "flops": n * 8 / 7 * 400}
    res = 3500.0 if sst else (1300.0 if kind == "box" else 2100.0)
    met = 20 if sst else (13 if kind == "box" else 19)
    if kind == "residual":
        return {"bytes": 8 * n * (2 * nv + met), "flops": n * res}
    imp = 700.0 if sst else 450.0
    cyc = c.get("cycles", 1)
    if c.get("levels", 1) > 1:
        return {"bytes": 8 * n * (2 * nv + met) * cyc * 8 / 7, "flops": n * cyc * (2 * res + imp) * 8 / 7}
    return {"bytes": 8 * n * (2 * nv + met) * cyc, "flops": n * cyc * (res + imp)}


def tolerance(c):
    """FP64 sums in another order: a restatement without fused multiply-adds
    differs by up to 5e-14 in a small velocity component after a few cycles
    and by 2e-12 in the wall-normal residual, a difference of nearly equal
    pressures; longer calls and thinner cells amplify that.  The FP32
    implicit stage: the FP64 one differs from it by up to 3e-5 in a velocity
    component that the increments alone make.  BF16 operands in training."""
    if c["kind"] == "setup":
        return "exact"
    if c["kind"] == "train":
        return {"rel": 1e-2, "max": 0.5}
    if c["kind"] == "residual":
        return {"rel": 1e-11, "max": 1e-8}
    if c.get("fp32"):
        return {"rel": 1e-4, "max": 1e-3}
    return {"rel": 1e-11, "max": 1e-9}


# ---- the same in plain torch, 64 bits ----------------------------------------

def exact(c, seed):
    """The residual stage, a training step, and centres and wall distance of
    a set-up.  The other kinds iterate in 64 bits themselves: a restatement
    of a whole implicit cycle in 64 bits says no more than tolerance() does."""
    if c["kind"] == "residual":
        s = prepare(c, seed)
        g = s["g"]
        blk, prm = g.blocks[s["bid"]]
        shape = (blk.kmax + 4, blk.jmax + 4, blk.imax + 4)
        g.sync()
        a = {n: t.clone().view(shape) for n, t in _slots(g, s["bid"], SLOT).items()}
        g.close()
        out = _residual64(a, prm, blk.patches[0], bool(c["sst"]))
        return {n: t.reshape(-1) for n, t in out.items()}
    if c["kind"] == "train":
        return _train64(prepare(c, seed))
    if c["kind"] == "setup" and c["ni"] * c["nj"] * c["nk"] <= 600000:
        return _setup64(prepare(c, seed))
    return None


def _setup64(s):
    c = s["case"]
    names = grid.METRIC_NAMES + ("DISTW",)
    ng = 2
    P = [torch.as_tensor(x, device="cuda") for x in s["nodes"]]
    for ax in range(3):   # mirror reflection of the nodes, layer by layer
        Q = []
        for a in P:
            n = a.shape[ax]
            sel = lambda i: a.narrow(ax, i, 1)  # noqa: B023,E731
            Q.append(torch.cat([2 * sel(0) - sel(m) for m in range(ng, 0, -1)] + [a] +
                               [2 * sel(n - 1) - sel(n - 1 - m) for m in range(1, ng + 1)], dim=ax))
        P = Q
    for a in P:   # the first layer's edges and corners reflect diagonally
        n = [x - 2 * ng for x in a.shape]
        at = lambda ax, side: (ng - 1, ng, ng + 1) if side == 0 else (ng + n[ax], ng + n[ax] - 1, ng + n[ax] - 2)  # noqa: B023,E731
        for u, v in ((0, 1), (0, 2), (1, 2)):
            w = 3 - u - v
            for su in (0, 1):
                for sv in (0, 1):
                    ix = [[None] * 3 for _ in range(3)]
                    for q in range(3):
                        ix[q][u], ix[q][v], ix[q][w] = at(u, su)[q], at(v, sv)[q], slice(ng, ng + n[w])
                    a[tuple(ix[0])] = 2.0 * a[tuple(ix[1])] - a[tuple(ix[2])]
        for k in range(8):
            p = [at(ax, (k >> ax) & 1) for ax in range(3)]
            a[p[0][0], p[1][0], p[2][0]] = 2.0 * a[p[0][1], p[1][1], p[2][1]] - a[p[0][2], p[1][2], p[2][2]]
    lo, hi = slice(None, -1), slice(1, None)
    cen = [sum(a[k, j, i] for k in (lo, hi) for j in (lo, hi) for i in (lo, hi)) / 8.0 for a in P]
    q = torch.stack([x.reshape(-1) for x in cen], dim=1)
    w = torch.as_tensor(np.ascontiguousarray(s["walls"]), device="cuda")
    best = torch.empty(q.shape[0], dtype=torch.float64, device="cuda")
    for i in range(0, q.shape[0], 8192):
        d2 = sum((q[i:i + 8192, None, x] - w[None, :, x]) ** 2 for x in range(3))
        best[i:i + 8192] = d2.min(dim=1).values.sqrt()
    got = {"XC": q[:, 0].contiguous(), "YC": q[:, 1].contiguous(), "ZC": q[:, 2].contiguous(), "DISTW": best}
    first = {n: got.get(n) for n in names}
    s["g"].close()
    return [first] + [{n: None for n in names} for _ in range(c["levels"] - 1)]


def _train64(s):
    net, x, t = s["net"], s["x"].double(), s["t"].double()
    w = net.w.double().clone().requires_grad_(True)
    h = x
    wt = lambda l: w[l.off:l.off + l.n * l.k].view(l.n, l.k)  # noqa: E731
    for l in net.L[:4]:
        h = h @ wt(l).T + w[l.boff:l.boff + l.n]
        h = torch.nn.functional.silu(h) if l.act else h
    h = h.reshape(-1, warmstart.CH)
    for l in net.L[4:]:
        h = h.reshape(-1, l.k) @ wt(l).T + w[l.boff:l.boff + l.n]
        h = torch.nn.functional.silu(h) if l.act else h
    loss = ((h[:, :t.shape[1]] - t) ** 2).mean()
    loss.backward()
    g = w.grad
    new = w.detach() - 2e-3 * g / (g.abs() + 1e-8)   # Adam's first step
    return {"pred": h.detach(), "loss": loss.detach().reshape(1), "grad": g, "w": new}


def _limited(q, inter):
    """The MUSCL pair of the face between q[1] and q[2]."""
    k1 = {1: 0.0, 3: 1.3333333}[inter]
    r1, r2 = 0.25 * k1, 0.25 * (2.0 - k1)
    d0, d1, d2 = q[1] - q[0], q[2] - q[1], q[3] - q[2]
    e = d1 * d1 + 1e-10
    return (q[2] - (e + d1 * d2) / (e + d2 * d2) * (d1 * r1 + d2 * r2),
            q[1] + (e + d1 * d0) / (e + d0 * d0) * (d1 * r1 + d0 * r2))


def _residual64(a, p, inl, sst):
    """The level-1 residual of a channel block (inlet at low i, outlet at high
    i, walls at low and high j, symmetry at both k) from its arrays."""
    mx = torch.clamp_min
    axis = {1: 2, 2: 1, 3: 0}

    def R(x, g=0, ax=None, o=0):   # the interior and g ghost layers, shifted by o along ax
        return x[tuple(slice(2 - g + (o if q == ax else 0), x.shape[q] - 2 + g + (o if q == ax else 0)) for q in range(3))]

    def wall(side, o):   # the cell layer o inside (negative: outside) of a wall, whole block interior
        n = a["U"].shape[1]
        return (slice(2, -2), 2 + o if side == 0 else n - 3 - o, slice(2, -2))

    def refcen():
        for side in (0, 1):
            b, l, t = wall(side, -1), wall(side, 0), wall(side, 1)
            ext = lambda n: 2.0 * a[n][l] - a[n][t]  # noqa: B023,E731
            a["RO"][b] = mx(ext("RO"), 0.001 * p.frsden)
            a["P"][b] = mx(ext("P"), 0.001 * p.frspre)
            for n in ("E", "U", "V", "W", "RM", "RN", "RW"):
                a[n][b] = ext(n)
            if sst:
                a["RK"][b] = mx(ext("RK"), p.rklim)
                a["REPS"][b] = mx(ext("REPS"), p.epslim)

    def gradient(f, g):   # volume gradient from distance-weighted face values
        pv = 0.5 / R(a["VOL"], g)
        out = [0.0, 0.0, 0.0]
        for d in (1, 2, 3):
            ax, D, A = axis[d], a["D%d" % d], a["A%d" % d]
            for o in (-1, 1):
                w1 = 2.0 * R(D, g) / (R(D, g) + R(D, g, ax, o))
                v = (2.0 - w1) * R(f, g) + w1 * R(f, g, ax, o)
                h = 0 if o < 0 else 1
                for x in range(3):
                    out[x] = out[x] + o * pv * R(A, g, ax, h) * R(a["A%d%sA" % (d, "XYZ"[x])], g, ax, h) * v
        return out

    def velocity_gradients():
        gu, gv, gw = (gradient(a[n], 1) for n in "UVW")
        gt = gradient(a["TEMP"], 1)
        for n, v in {"S11": gu[0], "S22": gv[1], "S33": gw[2], "S12": .5 * (gu[1] + gv[0]), "S13": .5 * (gu[2] + gw[0]),
                     "S23": .5 * (gv[2] + gw[1]), "W12": .5 * (gu[1] - gv[0]), "W13": .5 * (gu[2] - gw[0]),
                     "W23": .5 * (gv[2] - gw[1]), "DTDX": gt[0], "DTDY": gt[1], "DTDZ": gt[2]}.items():
            R(a[n], 1)[:] = v
        s2 = sum((2.0 if n in ("S12", "S13", "S23") else 1.0) * R(a[n], 1) ** 2 for n in
                 ("S11", "S12", "S13", "S22", "S23", "S33"))
        R(a["STRAIN"], 1)[:] = torch.sqrt(2.0 * s2)
        R(a["OHMI"], 1)[:] = 2.0 * torch.sqrt(sum(R(a[n], 1) ** 2 for n in ("W12", "W13", "W23")))

    if not sst:
        refcen()
        velocity_gradients()
    else:
        velocity_gradients()
        ro, rk, re, dw, vis = (R(a[n]) for n in ("RO", "RK", "REPS", "DISTW", "VIS"))
        om, kk, tiny = re / ro, mx(rk / ro, 0.0), 1e-20
        aux = vis / mx(re * dw * dw, tiny)
        f2 = torch.tanh(torch.maximum(2.0 * kk.sqrt() / mx(0.09 * om * dw, tiny), 500.0 * aux) ** 2)
        f3 = 1.0 - torch.tanh((150.0 * aux) ** 4)
        mut = torch.minimum(rk / om, 0.31 * rk / mx(R(a["STRAIN"]) * f2 * f3, tiny))
        mut = torch.minimum(mx(mut, 1e-3 * p.frsvis), p.turlim * vis)
        R(a["VIST"])[:] = mut
        R(a["EPS2"])[:] = 1.0 + mut / vis
        # cross diffusion (unweighted face averages)
        k_, o_ = a["RK"] / a["RO"], a["REPS"] / a["RO"]
        div = 0.0
        gk, go = [0.0] * 3, [0.0] * 3
        for d in (1, 2, 3):
            ax = axis[d]
            for o in (-1, 1):
                h = 0 if o < 0 else 1
                for x in range(3):
                    f = o * 0.5 / R(a["VOL"]) * R(a["A%d" % d], 0, ax, h) * R(a["A%d%sA" % (d, "XYZ"[x])], 0, ax, h)
                    gk[x] = gk[x] + f * (R(k_) + R(k_, 0, ax, o))
                    go[x] = go[x] + f * (R(o_) + R(o_, 0, ax, o))
        div = sum(x * y for x, y in zip(gk, go))
        cross = 2.0 * 0.856 * ro * div / om
        cdmin = 1e-8 * max(0.0, float(cross.max()))
        cd = mx(cross, cdmin)
        a13 = torch.maximum(kk.sqrt() / mx(0.09 * om * dw, tiny), 500.0 * aux)
        f1 = torch.tanh(torch.minimum(a13, 4.0 * 0.856 * rk / mx(cd * dw * dw, tiny)) ** 4)
        f1 = torch.where(dw < 0.40559e-7 * math.sqrt(p.re), torch.ones_like(f1), f1)
        R(a["FUN1"])[:] = f1
        refcen()
        prod = torch.minimum((R(a["EPS2"]) - 1.0) * vis * R(a["STRAIN"]) * R(a["OHMI"]), 20.0 * 0.09 * re * rk / ro)
        k_, o_ = a["RK"] / a["RO"], a["REPS"] / a["RO"]
        for x, (gx, gy) in enumerate(zip(gradient(k_, 1), gradient(o_, 1))):
            R(a["DKD" + "XYZ"[x]], 1)[:] = gx
            R(a["DED" + "XYZ"[x]], 1)[:] = gy

    # inlet (low i) and outlet (high i) ghosts
    J = (slice(2, -2), slice(2, -2))
    ii, g1, g2 = J + (2,), J + (1,), J + (0,)
    for gh in (g1, g2):
        for n in ("EPS2", "VIST", "P"):
            a[n][gh] = a[n][ii]
        a["TEMP"][gh] = inl.bount
        for n, b in (("U", inl.bounu), ("V", inl.bounv), ("W", inl.bounw)):
            a[n][gh] = b * inl.bounr / a["RO"][gh]
        if sst:
            a["RK"][gh], a["REPS"][gh] = inl.bounrk, inl.bounep
    ii, g1, g2 = J + (-3,), J + (-2,), J + (-1,)
    nrm = [a["A1%sA" % x][J + (-2,)] for x in "XYZ"]
    vel = 0.5 * sum(n * (a[v][ii] + b) for n, v, b in zip(nrm, "UVW", (inl.bounu, inl.bounv, inl.bounw)))
    turlim = p.turlim if sst else 1e-6
    eps2 = torch.clamp_max(a["EPS2"][ii], turlim)
    vist = torch.minimum(a["VIST"][ii], turlim * a["VIS"][g2])
    u_out = a["RO"][ii] * a["U"][ii] / a["RO"][g1]
    out = vel > 0.0
    if not bool(out.all()):
        raise ValueError("the restatement covers an outlet that flows out everywhere")
    for gh in (g1, g2):
        a["P"][gh] = inl.bounp
        a["EPS2"][gh], a["VIST"][gh] = eps2, vist
        a["U"][gh], a["V"][gh], a["W"][gh] = u_out, a["V"][ii], a["W"][ii]
        a["TEMP"][gh] = a["TEMP"][ii]
        if sst:
            a["RK"][gh], a["REPS"][gh] = a["RK"][ii], a["REPS"][ii]

    total = 0.0
    for d in (3, 1, 2):
        fl = _face_fluxes(a, p, d, sst)
        n = fl.shape[1 + axis[d]] - 1
        total = total - (fl.narrow(1 + axis[d], 1, n) - fl.narrow(1 + axis[d], 0, n))
    total = total / R(a["VOL"])
    if sst:
        f1, of = R(a["FUN1"]), mx(1.0 - R(a["FUN1"]), 0.0)
        beta, sig = f1 * 0.075 + of * 0.0828, f1 * 0.5 + of * 0.856
        gam = beta / 0.09 - sig * 0.41 ** 2 / math.sqrt(0.09)
        re, rk, ro = R(a["REPS"]), R(a["RK"]), R(a["RO"])
        mut = mx(R(a["EPS2"]) - 1.0, 1e-10) * R(a["VIS"])
        total[5] += prod - 0.09 * rk * re / ro
        total[6] += of * cross + re * (gam * ro * prod / (mut * re) - beta * re / ro)
    names = RESID + (("DRK", "DEPS") if sst else ())
    res = {}
    for v, n in enumerate(names):
        full = torch.zeros_like(a["RO"])
        R(full)[:] = total[v]
        res[n] = full
    return res


def _face_fluxes(a, p, d, sst):
    """[nv, faces] of direction d: Roe with MUSCL, full viscous stresses, walls."""
    ax = {1: 2, 2: 1, 3: 0}[d]
    mx = torch.clamp_min

    def F(x, o=0):   # cell L + o of every face (L: its high side)
        return x[tuple(slice(2 + o, x.shape[q] - 1 + o) if q == ax else slice(2, -2) for q in range(3))]

    inter = (p.interi, p.interj, p.interk)[d - 1]
    nx, ny, nz = (F(a["A%d%sA" % (d, x)]) for x in "XYZ")
    area = F(a["A%d" % d])
    pair = lambda n, i: _limited([F(a[n], o) for o in (-2, -1, 0, 1)], i)  # noqa: E731
    lim = lambda pq, b: (mx(pq[0], b), mx(pq[1], b))  # noqa: E731
    roR, roL = lim(pair("RO", inter), 0.001 * p.frsden)
    (uR, uL), (vR, vL), (wR, wL) = pair("U", inter), pair("V", inter), pair("W", inter)
    pR, pL = lim(pair("P", inter), 0.001 * p.frspre)
    kR = kL = eR_ = eL_ = torch.zeros_like(pR)
    if sst:
        kR, kL = lim(pair("RK", 1), 0.001 * p.rklim)
        eR_, eL_ = lim(pair("REPS", 1), 0.001 * p.epslim)
    gm = 1.0 / (p.gamma - 1.0)
    eR, eL, eLR, eRL = pR * gm / roR, pL * gm / roL, pR * gm / roL, pL * gm / roR
    o2 = 0 if d == 3 else -1
    dp_, dr_ = 0.0, 0.0
    for o in (0, o2):
        rp, rh, ro, pp = (F(a[n], o) for n in ("DRDP", "DRDH", "RO", "P"))
        dp_ = dp_ + 0.5 * (-rp / rh - 1.0 / ro)
        dr_ = dr_ + 0.5 * (1.0 / rh + pp / ro ** 2)
    big = (2.0 * (pR - pL)).abs() >= 1e-2 * (pR + pL)
    dedp = torch.where(big, (eR + eLR - eL - eRL) / torch.where(big, 2.0 * (pR - pL), 1.0), dp_)
    big = (2.0 * (roR - roL)).abs() >= 1e-2 * (roR + roL)
    dedr = torch.where(big, (eR + eRL - eL - eLR) / torch.where(big, 2.0 * (roR - roL), 1.0), dr_)
    ur, ul = nx * uR + ny * vR + nz * wR, nx * uL + ny * vL + nz * wL
    tR = [uR - ur * nx, vR - ur * ny, wR - ur * nz]
    tL = [uL - ul * nx, vL - ul * ny, wL - ul * nz]
    c23 = 0.6667
    rkR, rkL, omR, omL = kR / roR, kL / roL, eR_ / roR, eL_ / roL
    hR = eR + 0.5 * (uR ** 2 + vR ** 2 + wR ** 2) + rkR + pR / roR
    hL = eL + 0.5 * (uL ** 2 + vL ** 2 + wL ** 2) + rkL + pL / roL
    rh = torch.sqrt(roR * roL)
    cl = roL / (roL + rh)
    mean = lambda x, y: (1.0 - cl) * x + cl * y  # noqa: E731
    uh, hh, eh, kh, oh = mean(ur, ul), mean(hR, hL), mean(eR, eL), mean(rkR, rkL), mean(omR, omL)
    th = [mean(x, y) for x, y in zip(tR, tL)]
    ph = rh * (hh - eh - 0.5 * (uh ** 2 + sum(x * x for x in th)) - kh)
    ph = torch.maximum(torch.minimum(torch.maximum(pR, pL), ph), torch.minimum(pR, pL))
    drdh = 1.0 / (dedr - ph / rh ** 2)
    drdp = -drdh * (dedp + 1.0 / rh)
    c2 = (1.0 + c23 * kh / rh * drdp) / (drdh / rh + drdp)
    cR, cL = F(a["C"]), F(a["C"], -1)
    c2 = torch.maximum(torch.minimum(torch.maximum(cR, cL) ** 2, c2), torch.minimum(cR, cL) ** 2)
    ch = torch.sqrt(c2)
    dro, du, dk = roR - roL, ur - ul, rkR - rkL
    dp = pR - pL + c23 * (kh * dro + rh * dk)
    a1, a2, a3 = 0.5 * (dp + rh * ch * du) / c2, 0.5 * (dp - rh * ch * du) / c2, dro - dp / c2
    l1, l2, l3 = (uh + ch).abs(), (uh - ch).abs(), uh.abs()
    mR, mL = roR * ur, roL * ul
    damp, dc = l1 * a1 + l2 * a2 + l3 * a3, l1 * a1 - l2 * a2
    ha = 0.5 * area
    fn = ha * (mR * ur + pR + c23 * kR + mL * ul + pL + c23 * kL - (damp * uh + dc * ch))
    ft = [ha * (mR * x + mL * y - damp * z - l3 * rh * (x - y)) for x, y, z in zip(tR, tL, th)]
    tj = l3 * rh * sum((x - y) * z for x, y, z in zip(tR, tL, th))
    f5 = ha * (mR * (hR + c23 * kR / roR) + mL * (hL + c23 * kL / roL) - damp * hh -
               (dc * uh * ch - l3 * a3 * rh * c2 * dedp + tj) + l3 * rh * dk * (1.0 - c23 * rh * dedp))
    f = [ha * (mR + mL - damp), nx * fn + ft[0], ny * fn + ft[1], nz * fn + ft[2], f5]
    if sst:
        f += [ha * (mR * rkR + mL * rkL - damp * kh - l3 * rh * dk),
              ha * (mR * omR + mL * omL - damp * oh - l3 * rh * (omR - omL))]

    # viscous part
    D = a["D%d" % d]
    w1 = 2.0 * F(D) / (F(D) + F(D, -1))
    at = lambda n: 0.5 * ((2.0 - w1) * F(a[n]) + w1 * F(a[n], -1))  # noqa: E731
    s = [F(a[n]) - F(a[n], -1) for n in ("XC", "YC", "ZC")]
    ln = torch.sqrt(sum(x * x for x in s)) + 1e-21
    sx, sy, sz = (x / ln for x in s)
    S = {n: at(n) for n in ("S11", "S12", "S13", "S22", "S23", "S33", "W12", "W13", "W23", "DTDX", "DTDY", "DTDZ")}
    gu = [S["S11"], S["S12"] + S["W12"], S["S13"] + S["W13"]]
    gv = [S["S12"] - S["W12"], S["S22"], S["S23"] + S["W23"]]
    gw = [S["S13"] - S["W13"], S["S23"] - S["W23"], S["S33"]]
    al = sx * nx + sy * ny + sz * nz
    pos = al > 0.0
    surf = 0.5 * area * sum(F(a["EPS2"], o) * F(a["VIS"], o) for o in (0, -1))
    sure = 0.5 * area * sum(F(a["CP"], o) * F(a["VIST"], o) / p.prt + F(a["CH"], o) for o in (0, -1))
    along = lambda g: g[0] * sx + g[1] * sy + g[2] * sz  # noqa: E731
    du_, dv_, dw_ = (F(a[n]) - F(a[n], -1) for n in "UVW")
    corr = (nx * du_ + ny * dv_ + nz * dw_) / ln - (nx * along(gu) + ny * along(gv) + nz * along(gw))
    base = [2.0 * (nx * S["S11"] + ny * S["S12"] + nz * S["S13"]), 2.0 * (nx * S["S12"] + ny * S["S22"] + nz * S["S23"]),
            2.0 * (nx * S["S13"] + ny * S["S23"] + nz * S["S33"])]
    div = 0.6666667 * (gu[0] + gv[1] + gw[2])
    t = []
    for b, q, g, sd, nd in zip(base, (du_, dv_, dw_), (gu, gv, gw), (sx, sy, sz), (nx, ny, nz)):
        b = torch.where(pos, al * (q / ln - along(g)) + sd * corr + b, b)
        t.append(surf * (b - nd * div))
    heat = sure * (S["DTDX"] * nx + S["DTDY"] * ny + S["DTDZ"] * nz)
    q5 = 0.5 * sum((F(a[n]) + F(a[n], -1)) * x for n, x in zip("UVW", t)) + heat
    slope = (F(a["TEMP"]) - F(a["TEMP"], -1)) / ln - (sx * S["DTDX"] + sy * S["DTDY"] + sz * S["DTDZ"])
    q5 = torch.where(pos, sure * al * slope + q5, q5)
    for v in range(3):
        f[1 + v] = f[1 + v] - t[v]
    f[4] = f[4] - q5
    if sst:
        f1 = F(a["FUN1"])
        of = mx(1.0 - f1, 0.0)
        vv, vt = F(a["VIS"]) + F(a["VIS"], -1), F(a["VIST"]) + F(a["VIST"], -1)
        ap = mx(al, 0.0)
        for v, (n, g, sig) in enumerate((("RK", "DKD", f1 * 0.85 + of), ("REPS", "DED", f1 * 0.5 + of * 0.856))):
            jump = F(a[n]) / F(a["RO"]) - F(a[n], -1) / F(a["RO"], -1)
            diff = -0.5 * area * (vv + vt * sig) * (ap * jump / ln + at(g + "X") * (nx - ap * sx) + at(g + "Y") * (ny - ap * sy) +
                                                    at(g + "Z") * (nz - ap * sz))
            f[5 + v] = f[5 + v] + diff
            if v == 0:
                f[4] = f[4] + diff
    fl = torch.stack(f)
    if d == 2:
        for side in (0, 1):
            fl[:, :, 0 if side == 0 else -1, :] = _wall_fluxes(a, p, side, inter, sst)
    return fl


def _wall_fluxes(a, p, side, inter, sst):
    mx = torch.clamp_min
    n = a["U"].shape[1]
    sg = 1.0 if side == 0 else -1.0
    at = lambda x, j: a[x][2:-2, j, 2:-2]  # noqa: E731
    c1, c2 = (2, 3) if side == 0 else (n - 3, n - 4)
    fw, fi = (2, 3) if side == 0 else (n - 2, n - 3)
    ext = lambda x: 1.5 * at(x, c1) - 0.5 * at(x, c2)  # noqa: E731
    af = at("A2", fw)
    dist = (af + at("A2", fi)) / at("VOL", c1)
    sur = -dist * 0.166666667
    vis = mx(ext("VIS"), 0.01 * p.frsvis)
    pb = mx(ext("P"), 0.01 * p.frspre)
    nrm = [at("A2%sA" % x, fw) for x in "XYZ"]
    q = [sg * (9.0 * at(x, c1) - at(x, c2)) for x in "UVW"]
    div = 0.33333 * sum(x * y for x, y in zip(nrm, q))
    f = [torch.zeros_like(af)] + [af * (x * pb + sur * vis * (y + x * div)) for x, y in zip(nrm, q)] + [torch.zeros_like(af)]
    if sst:
        st = mx(ext("STRAIN"), 1e-3)
        nu = vis / mx(ext("RO"), 0.001 * p.frsden)
        yp = 2.0 * torch.sqrt(nu * st) / nu / dist
        sk = mx(torch.clamp_max(2.4 * yp ** 0.85, 8.0), 1e-3)
        om = st * torch.maximum(2500.0 / sk ** 2, 100.0 / sk)
        ev = sg * (9.0 * at("REPS", c1) / at("RO", c1) - at("REPS", c2) / at("RO", c2) - 8.0 * om)
        kv = sg * mx(9.0 * at("RK", c1) / at("RO", c1) - at("RK", c2) / at("RO", c2), 0.0)
        f6, f7 = af * sur * vis * kv, af * sur * vis * ev
        f[4] = f6
        f += [f6, f7]
    return torch.stack(f)
