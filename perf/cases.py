"""Workloads of the search path, each one pass through the package's public entry points.

A case is a dict of plain values.  ``listed()`` names the standing ones, ``draw(rng)`` gives another of the
same ranges, ``prepare(case, seed)`` makes the inputs and the objects a program keeps between calls,
``run(state)`` is one pass, ``work(case)`` the bytes and operations the path cannot do without, and
``exact(case, seed)`` the same outputs in 64 bits from plain numpy and torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from cpp_projects_b200 import CFdmtGpu, cluster, search, synth
from cpp_projects_b200.autograd import boxcar_snr, fdmt
from cpp_projects_b200.chunk import CChunk_gpu
from cpp_projects_b200.fdmt import FDMTGPU
from cpp_projects_b200.pipeline import BatchedSearch, BeamShape, device_filterbank

FMIN, FMAX = 1200.0, 1600.0        # the band of the repository's filterbank workloads (MHz)
TSAMP = 0.25e-6                    # coarse sample time of the voltage workloads (s)
PRECISIONS = {"f32": 0, "f16": 1, "bf16": 2}
MOST = 4096 * 131072               # channel samples of the largest case
ROOM = 1 << 24                     # candidates a program keeps room for


def _fdmt(name, nchan, ncols, max_dt, plan, precision="f32"):
    return {"name": name, "kind": "fdmt", "nchan": nchan, "ncols": ncols, "max_dt": max_dt, "plan": plan,
            "precision": precision}


def listed() -> list[dict]:
    return [
        # a receiver's short block through a plan made once: latency and launches
        _fdmt("fdmt_64x1000", 64, 1000, 64, "default"),
        # the single-beam workload (512 x 32768, max delay 512), the reference's constructor and call
        _fdmt("fdmt_512x32768", 512, 32768, 512, "default"),
        # a wide beam of the uneven set: odd length, so no row but the first is 16-byte aligned; tuned plan
        _fdmt("fdmt_4096x45001", 4096, 45001, 4096, "tuned"),
        # the reduced-precision workload (4096 x 2^17, 16-bit planes)
        _fdmt("fdmt_f16_4096x131072", 4096, 131072, 4096, "tuned", "f16"),
        # the reference's second FDMT variant on one of the search shapes
        {"name": "pravir_1024x16749", "kind": "pravir", "nchan": 1024, "ncols": 16749, "max_dt": 1024},
        # gradient of a DM-time plane with respect to the filterbank, as a user's own backward calls it
        {"name": "adjoint_256x24485", "kind": "adjoint", "nchan": 256, "ncols": 24485, "max_dt": 256},
        # one optimisation step of per-channel weights: forward, S/N at the pulses, backward
        {"name": "weights_step_1024x65536", "kind": "step", "nchan": 1024, "ncols": 65536, "max_dt": 1024},
        # detection and clustering of one beam's plane (row statistics, widths 1..32, three passes)
        {"name": "search_512x32768", "kind": "search", "rows": 512, "cols": 32768, "param": 5, "thr": 7.0},
        # the candidate step of a coherent chunk: normalised plane, every width up to 4
        {"name": "heap_1024x65536", "kind": "heap", "rows": 1024, "cols": 65536, "param": 4, "thr": 7.0},
        # a batch of uneven beams (the first 12 of the 48-beam workload) through the batched form
        {"name": "beams_12", "kind": "beams", "shapes": 2, "nbeams": 12},
        # one GUPPI chunk of 32 coarse channels, 2^20-point segments, 32 fine channels each
        {"name": "chunk_32x4x2e20", "kind": "chunk", "npol": 4, "nchan": 32, "len_sft": 32, "nbin": 1 << 20,
         "nfft": 4, "noverlap": 8192, "max_dt": 1024, "dm": 56.8},
        # a short chunk of another geometry (library FFT sizes), one polarisation pair
        {"name": "chunk_16x2x2e16", "kind": "chunk", "npol": 4, "nchan": 16, "len_sft": 16, "nbin": 1 << 16,
         "nfft": 2, "noverlap": 1024, "max_dt": 256, "dm": 20.0},
    ]


def _between(rng: random.Random, lo: int, hi: int) -> int:
    """A whole number between lo and hi, even over the logarithm; odd ones as likely as even ones."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["fdmt"] * 4 + ["pravir", "adjoint", "step", "search", "search", "heap", "beams", "chunk"])
    if kind in ("fdmt", "pravir", "adjoint", "step"):
        nchan = rng.choice([64, 96, 128, 256, 256, 512, 512, 1024, 1024, 2048, 4096] if kind == "fdmt"
                           else [64, 128, 256, 512, 1024])
        most = 131072 if kind == "fdmt" else 65536
        ncols = _between(rng, max(1000, 2 * nchan), most)
        case = {"kind": kind, "nchan": nchan, "ncols": ncols, "max_dt": nchan}
        if kind == "fdmt":
            case["max_dt"] = rng.choice([nchan] * 4 + [nchan // 2, 3 * nchan // 2])
            case["max_dt"] = min(case["max_dt"], MOST // ncols)
            case["plan"] = rng.choice(["default", "default", "tuned"])
            case["precision"] = rng.choice(["f32"] * 5 + ["f16", "bf16"])
        return case
    if kind == "search":
        rows = rng.choice([128, 256, 512, 1024, 4096])
        return {"kind": kind, "rows": rows, "cols": _between(rng, 2048, 131072 if rows < 4096 else 65536),
                "param": rng.choice([4, 5, 5, 5, 6]), "thr": rng.choice([6.5, 7.0, 8.0])}
    if kind == "heap":
        rows = rng.choice([128, 256, 512, 1024])
        return {"kind": kind, "rows": rows, "cols": _between(rng, 2048, 131072), "param": rng.choice([2, 4, 4, 8]),
                "thr": rng.choice([6.5, 7.0, 8.0])}
    if kind == "beams":
        case = {"kind": kind, "shapes": rng.randrange(3, 10000), "nbeams": rng.randint(2, 6)}
        while case["nbeams"] > 1 and work(case)["bytes"] > 18e9:   # within the listed batch's size
            case["nbeams"] -= 1
        return case
    if rng.random() < 0.5:   # the 2^20-point geometry
        return {"kind": "chunk", "npol": rng.choice([2, 4, 4]), "nchan": rng.choice([4, 8, 16, 24]), "len_sft": 32,
                "nbin": 1 << 20, "nfft": rng.randint(1, 4), "noverlap": rng.choice([4096, 8192, 16384]),
                "max_dt": rng.choice([256, 512, 1024]), "dm": rng.uniform(5.0, 80.0)}
    nbin = 1 << rng.randint(13, 18)
    return {"kind": "chunk", "npol": rng.choice([2, 4]), "nchan": rng.choice([4, 8, 16, 32]),
            "len_sft": rng.choice([8, 16, 32]), "nbin": nbin, "nfft": rng.randint(1, 4), "noverlap": nbin // 64,
            "max_dt": rng.choice([64, 128, 256]), "dm": rng.uniform(1.0, 40.0)}


# ---- inputs ---------------------------------------------------------------------
def _device() -> torch.device:
    return torch.device("cuda", torch.cuda.current_device())


def _pulses(nchan, ncols, max_dt, seed, count=3) -> list:
    """Pulses of the filterbank workloads: width 1-32, amplitude 1.5-4, delay 10-90 % of the largest."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        span = float(rng.uniform(0.1, 0.9) * (max_dt - 1))
        width, amp = int(rng.integers(1, 33)), float(rng.uniform(1.5, 4.0)) / math.sqrt(max(1.0, nchan / 256))
        out.append(synth.Pulse(int(rng.integers(0, max(1, ncols - int(span) - width))), span, width, amp))
    return out


def _filterbank(nchan, ncols, max_dt, seed, count=3):
    pulses = _pulses(nchan, ncols, max_dt, seed, count)
    return device_filterbank(nchan, ncols, FMIN, FMAX, seed, pulses, _device()), pulses


def _plan(case, **kw):
    fuse = -2 if case.get("plan") == "tuned" else -1
    return CFdmtGpu(FMIN, FMAX, case["nchan"], case["ncols"], case["max_dt"], fuse_depth=fuse,
                    precision=PRECISIONS[case.get("precision", "f32")], **kw)


def _plane(rows, cols, seed) -> torch.Tensor:
    """The DM-time plane of a filterbank with `rows` channels and pulses in it."""
    x, _ = _filterbank(rows, cols, rows, seed)
    return CFdmtGpu(FMIN, FMAX, rows, cols, rows)(x)


def _beams(case):
    return synth.config2(seed=case["shapes"], nbeams=case["nbeams"], max_nchan=4096)


def _chunk_band(case):
    return 1200.0, 1200.0 + 4.0 * case["nchan"]


def _raw(case, seed):
    """int8 voltages: uniform noise in [-8, 7], a few samples of a strong broadband burst."""
    n = (case["nbin"] - 2 * case["noverlap"]) * case["nfft"]
    g = torch.Generator(device=_device()).manual_seed(int(seed))
    raw = torch.randint(-8, 8, (case["nchan"], n, case["npol"]), generator=g, device=_device(), dtype=torch.int8)
    t = int(np.random.default_rng(seed).integers(0, n - 64))
    raw[:, t: t + 4] = 7
    return raw


def prepare(case: dict, seed: int) -> dict:
    kind, dev = case["kind"], _device()
    if kind == "fdmt":
        x, _ = _filterbank(case["nchan"], case["ncols"], case["max_dt"], seed)
        return {"kind": kind, "x": x, "plan": _plan(case),
                "out": torch.empty((case["max_dt"], case["ncols"]), device=dev)}
    if kind == "pravir":
        x, _ = _filterbank(case["nchan"], case["ncols"], case["max_dt"], seed)
        plan = FDMTGPU(FMIN, FMAX, case["nchan"], case["ncols"], 1e-3, case["max_dt"])
        return {"kind": kind, "x": x, "plan": plan, "out": torch.empty((plan.out_rows, case["ncols"]), device=dev)}
    if kind == "adjoint":
        g = torch.Generator(device=dev).manual_seed(int(seed))
        gy = torch.randn((case["max_dt"], case["ncols"]), generator=g, device=dev)
        return {"kind": kind, "gy": gy, "plan": _plan(case),
                "gx": torch.empty((case["nchan"], case["ncols"]), device=dev)}
    if kind == "step":
        x, pulses = _filterbank(case["nchan"], case["ncols"], case["max_dt"], seed, count=8)
        return {"kind": kind, "x": x, "plan": _plan(case), "cells": _cells(case, pulses),
                "w": torch.ones(case["nchan"], device=dev, requires_grad=True)}
    if kind in ("search", "heap"):
        plane = _plane(case["rows"], case["cols"], seed)
        s = {"kind": kind, "case": dict(case), "plane": plane, "thr": torch.tensor([case["thr"]], device=dev),
             "cands": torch.zeros((ROOM, 4), dtype=torch.int32, device=dev)}
        if kind == "heap":
            s["plane"], _ = search.norm_rows(plane)
        for k in ("perm", "offsets", "delegates"):   # the program's own record of what was found
            s[k] = torch.zeros(ROOM + 1, dtype=torch.int32, device=dev)
        return s
    if kind == "beams":
        beams = _beams(case)
        x = [device_filterbank(b.nchan, b.nsamp, b.fmin, b.fmax, 1000 * seed + i,
                               _pulses(b.nchan, b.nsamp, b.max_dt, 1000 * seed + i, i % 4), dev)
             for i, b in enumerate(beams)]
        shapes = [BeamShape(b.nchan, b.nsamp, b.fmin, b.fmax, b.max_dt) for b in beams]
        return {"kind": kind, "x": x, "batch": BatchedSearch(shapes, capacity=1 << 25),
                "delegates": np.zeros((1 << 14, 4), np.int32), "sizes": np.zeros(1 << 14, np.int64)}
    fmin, fmax = _chunk_band(case)
    ch = CChunk_gpu(fmin, fmax, case["npol"], case["nchan"], case["len_sft"], 0, 0, case["dm"], 0.0, 1, 7.0, 1,
                    case["nbin"], case["nfft"], case["noverlap"], TSAMP, max_dt=case["max_dt"], dms=[case["dm"]])
    return {"kind": kind, "chunk": ch, "raw": _raw(case, seed), "spec": ch.complex_buffer(dev)}


def _cells(case, pulses) -> list:
    """{row, start, width} of each pulse: it reaches the lowest channel `span` samples after t0."""
    out = []
    for p in pulses:
        start = min(case["ncols"] - p.width, int(p.t0 + p.span))
        out.append([min(case["max_dt"] - 1, int(p.span)), start, p.width])
    return out


# ---- one pass -------------------------------------------------------------------
def _keep(s, cl):
    for k in ("perm", "offsets", "delegates"):
        v = getattr(cl, k)
        s[k][: v.shape[0]].copy_(v)
    return {k: s[k] for k in ("cands", "perm", "offsets", "delegates")}


def run(s: dict):
    kind = s["kind"]
    if kind == "fdmt":
        s["plan"].process_image(s["x"], s["out"])
        return s["out"]
    if kind == "pravir":
        s["plan"].execute(s["x"], s["x"].numel(), s["out"], s["out"].numel())
        return s["out"]
    if kind == "adjoint":
        return s["plan"].adjoint(s["gy"], s["gx"])
    if kind == "step":
        s["w"].grad = None
        y = fdmt(s["w"][:, None] * s["x"], s["plan"])
        snr = boxcar_snr(y, s["cells"])
        (-snr.sum()).backward()
        return {"plane": y.detach(), "snr": snr.detach(), "grad": s["w"].grad}
    if kind == "search":
        c = s["case"]
        st = search.row_stats(s["plane"])
        cands, n = search.boxcar_gather(s["plane"], c["thr"], 0, c["param"], stats=st, out=s["cands"])
        return {"stats": st, "found": n, **_keep(s, cluster.complete_clusterization(cands, (16, 8, 1 << 30)))}
    if kind == "heap":
        c = s["case"]
        cands, n = search.gather_candidates_in_heap_with_plan(s["plane"], c["rows"], c["cols"], s["thr"], c["param"],
                                                              out=s["cands"])
        return {"found": n, **_keep(s, cluster.complete_clusterization(cands, (2, 1, 2)))}
    if kind == "beams":
        got = s["batch"].run(s["x"])
        at = 0
        for r in got:
            k = len(r.delegates)
            s["delegates"][at: at + k] = r.delegates.view(np.int32).reshape(-1, 4)
            s["sizes"][at: at + k] = r.group_sizes
            at += k
        return {"found": np.array([[r.n_candidates, len(r.delegates)] for r in got], np.int64),
                "delegates": s["delegates"], "sizes": s["sizes"]}
    planes = s["chunk"].process_raw(s["raw"], s["spec"])
    return {"planes": planes, "spectra": s["spec"]}


# ---- work -----------------------------------------------------------------------
def _tree(nchan, ncols, max_dt):
    """Adds of the transform, one per merged row and sample (about max_dt + nchan / 2^l rows a level)."""
    return ncols * sum(max_dt + (nchan >> l) for l in range(1, max(1, (nchan - 1).bit_length()) + 1))


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("fdmt", "pravir", "adjoint", "step"):
        n, t, d = case["nchan"], case["ncols"], case["max_dt"]
        io, ops = 4 * (n + d) * t, _tree(n, t, d)
        if kind == "step":   # input, plane and both gradients once each
            return {"bytes": 2 * io, "flops": 2 * ops + 6 * n * t}
        return {"bytes": io, "flops": ops}
    if kind == "search":     # statistics need a whole row before its first test: two reads
        n = case["rows"] * case["cols"]
        return {"bytes": 8 * n, "flops": n * (5 + (1 << case["param"]))}
    if kind == "heap":
        n = case["rows"] * case["cols"]
        return {"bytes": 4 * n, "flops": n * 2 * case["param"]}
    if kind == "beams":
        w = {"bytes": 0, "flops": 0}
        for b in _beams(case):
            n = b.max_dt * b.nsamp
            w["bytes"] += 4 * b.nchan * b.nsamp + 4 * n + 8 * n
            w["flops"] += _tree(b.nchan, b.nsamp, b.max_dt) + 37 * n
        return w
    pol, n = case["npol"] // 2, case["nchan"] * case["nfft"] * case["nbin"]
    rows, msamp = case["nchan"] * case["len_sft"], case["nfft"] * (case["nbin"] - 2 * case["noverlap"]) // case["len_sft"]
    fft = 5 * pol * n * (math.log2(case["nbin"]) + math.log2(case["nbin"] // case["len_sft"]))
    return {"bytes": 2 * pol * n + 8 * pol * n + 4 * case["max_dt"] * msamp,
            "flops": fft + _tree(rows, msamp, case["max_dt"])}


# ---- the same in 64 bits ----------------------------------------------------------
def _f32(v):
    return np.float32(v)


def _keith_plan(fmin, fmax, nchan, max_dt):
    """(level-0 rows per channel, [(tail row, head row or -1, shift)] per level): float edges squared in
    float, reciprocals and differences in double, truncated float products."""
    fmin, fmax = _f32(fmin), _f32(fmax)

    def inv(f):
        return 1.0 / float(_f32(f * f))

    def delta(f0, f1):
        return math.ceil((inv(f0) - inv(f1)) / (inv(fmin) - inv(fmax)) * (max_dt - 1.0))

    bw = _f32(fmax - fmin)
    r0 = delta(fmin, _f32(fmin + _f32(bw / _f32(nchan)))) + 1
    freq = [_f32(fmin + _f32(_f32(_f32(i) * bw) / _f32(nchan))) for i in range(nchan)] + [fmax]
    rows, levels = [r0] * nchan, []
    while len(rows) > 1:
        cum = np.concatenate([[0], np.cumsum(rows)])
        nrows, nfreq, a, b, s = [], [], [], [], []
        for i in range(0, len(rows) - 1, 2):
            lo, mid, hi = freq[i], freq[i + 1], freq[i + 2]
            n = delta(lo, hi) + 1
            whole = _f32(inv(lo) - inv(hi))
            c0, c1 = _f32(_f32(inv(lo) - inv(mid)) / whole), _f32(_f32(inv(mid) - inv(hi)) / whole)
            j = np.arange(n, dtype=np.float32)
            j0, j1 = (c0 * j).astype(np.int64), (c1 * j).astype(np.int64)
            a.append(cum[i] + j0), b.append(cum[i + 1] + j1), s.append(j0)
            nrows.append(n), nfreq.append(lo)
        if len(rows) % 2:   # the last sub-band goes up as it is
            n = rows[-1]
            a.append(cum[-2] + np.arange(n)), b.append(np.full(n, -1)), s.append(np.zeros(n, np.int64))
            nrows.append(n), nfreq.append(freq[len(rows) - 1])
        levels.append((np.concatenate(a), np.concatenate(b), np.concatenate(s)))
        rows, freq = nrows, nfreq + [fmax]
    return r0, levels


def _merge(p, level):
    """out[g][t] = p[tail][t] + p[head][t - shift] (from sample `shift` on)."""
    a, b, s = level
    out = p[torch.from_numpy(a).to(p.device)]
    for sh in np.unique(s[b >= 0]):
        g = np.nonzero((b >= 0) & (s == sh))[0]
        gi, bi = torch.from_numpy(g).to(p.device), torch.from_numpy(b[g]).to(p.device)
        out[gi, sh:] += p[bi, : p.shape[1] - sh]
    return out


def _merge_adjoint(g, level, rows):
    a, b, s = level
    out = torch.zeros((rows, g.shape[1]), dtype=g.dtype, device=g.device)
    out.index_add_(0, torch.from_numpy(a).to(g.device), g)
    for sh in np.unique(s[b >= 0]):
        k = np.nonzero((b >= 0) & (s == sh))[0]
        out[:, : g.shape[1] - sh].index_add_(0, torch.from_numpy(b[k]).to(g.device),
                                             g[torch.from_numpy(k).to(g.device), sh:].contiguous())
    return out


def _fdmt64(x, r0, levels):
    """x: nchan x T float64; level-0 row r of a channel is the mean of x[t-r .. t], 0 before sample r."""
    n, t = x.shape
    p = torch.zeros((n, r0, t), dtype=torch.float64, device=x.device)
    run = torch.zeros_like(x)
    for r in range(r0):
        run[:, r:] += x[:, : t - r]
        p[:, r, r:] = run[:, r:] / (r + 1)
    del run
    p = p.reshape(n * r0, t)
    for level in levels:
        p = _merge(p, level)
    return p


def _fdmt64_adjoint(gy, nchan, r0, levels):
    rows = [nchan * r0] + [len(lv[0]) for lv in levels]
    g = gy
    for k in range(len(levels) - 1, -1, -1):
        g = _merge_adjoint(g, levels[k], rows[k])
    t = g.shape[1]
    g = g.reshape(nchan, r0, t)
    out = torch.zeros((nchan, t), dtype=torch.float64, device=g.device)
    for r in range(r0):
        for j in range(r + 1):   # x[t - j] is in the mean of row r at samples t >= r
            out[:, r - j: t - j] += g[:, r, r:] / (r + 1)
    return out


def _pravir64(x, max_dt):
    """The other variant: delay grids 0..rounded span per sub-band, window means, rounded mid-band shifts."""
    n, t = x.shape
    fmin, fmax = _f32(FMIN), _f32(FMAX)

    def power(f):
        return _f32(float(f) ** -2.0)

    def cff(a, b, c, d):
        return _f32(_f32(power(a) - power(b)) / _f32(power(c) - power(d)))

    def rnd(v):
        return int(math.floor(abs(float(v)) + 0.5) * (1 if v >= 0 else -1))

    def grid(fs, fe):
        return list(range(0, rnd(_f32(_f32(max_dt) * cff(fs, fe, fmin, fmax))) + 1))

    df = _f32(_f32(fmax - fmin) / _f32(n))
    corr = _f32(df / _f32(2))
    grids = [grid(_f32(_f32(df * _f32(i)) + fmin), _f32(_f32(_f32(df * _f32(i)) + fmin) + df)) for i in range(n)]
    csum = torch.cat([torch.zeros((n, 1), dtype=torch.float64, device=x.device), x.cumsum(1)], 1)
    planes = []
    for c, g in enumerate(grids):
        for d in g:
            row = torch.zeros(t, dtype=torch.float64, device=x.device)
            row[d:] = (csum[c, d + 1:] - csum[c, : t - d]) / (d + 1)
            planes.append(row)
    p = torch.stack(planes)
    del csum, planes
    bot = df
    while len(grids) > 1:   # powers of two only: no sub-band is carried over
        bot2 = _f32(bot * _f32(2))
        cum = np.concatenate([[0], np.cumsum([len(g) for g in grids])])
        new, a, b, s = [], [], [], []
        for i in range(len(grids) // 2):
            fs = _f32(_f32(bot2 * _f32(i)) + fmin)
            fe, fm = _f32(fs + bot2), _f32(fs + _f32(bot2 / _f32(2)))
            cur = grid(fs, fe)
            k1, k2 = cff(fs, _f32(fm - corr), fs, fe), cff(fs, _f32(fm + corr), fs, fe)
            for d in cur:
                m1, m2 = rnd(_f32(_f32(d) * k1)), rnd(_f32(_f32(d) * k2))
                a.append(cum[2 * i] + min(m1, len(grids[2 * i]) - 1))
                b.append(cum[2 * i + 1] + max(0, min(d - m2, len(grids[2 * i + 1]) - 1)))
                s.append(m2)
            new.append(cur)
        p = _merge(p, (np.array(a), np.array(b), np.array(s)))
        grids, bot = new, bot2
    return p


def _chunk64(case, raw):
    """Unpack, segment FFTs, chirp, sub-band inverse FFTs, detection, dedispersion, preprocessing, transform."""
    dev, dm = raw.device, case["dm"]
    fmin, fmax = (_f32(v) for v in _chunk_band(case))
    nchan, sft, nbin, nfft, nov = case["nchan"], case["len_sft"], case["nbin"], case["nfft"], case["noverlap"]
    pol, mbin, n = case["npol"] // 2, nbin // sft, raw.shape[1]
    spec = torch.zeros((pol, nfft, nchan, nbin), dtype=torch.complex128, device=dev)
    for f in range(nfft):
        lo = (nbin - 2 * nov) * f - nov
        i0, i1 = max(0, lo), min(n, lo + nbin)
        part = raw[:, i0:i1].double()
        for q in range(pol):
            spec[q, f, :, i0 - lo: i1 - lo] = torch.complex(part[..., 2 * q], part[..., 2 * q + 1])
    for q in range(pol):
        spec[q] = torch.fft.fft(spec[q])
    bw = float(_f32(fmax - fmin))
    sub, fine = bw / nchan, bw / nchan / sft
    fb = -0.5 * fine + (torch.arange(mbin, dtype=torch.float64, device=dev) + 0.5) * fine / mbin
    taper = 1.0 / torch.sqrt(1.0 + (fb / (0.47 * fine)) ** 80)
    f0 = np.float32(float(fmin) + sub * (0.5 + np.arange(nchan)[:, None]) + fine * (np.arange(sft)[None] - sft / 2.0 + 0.5))
    f0 = torch.from_numpy(f0.astype(np.float64)).to(dev)[..., None]
    phase = dm * (fb / f0) * (fb / f0) / (f0 + fb) * 4.148808e9
    ang = -2.0 * math.pi * (phase - torch.trunc(phase))
    chirp = torch.polar((taper / nbin).expand_as(ang).contiguous(), ang).reshape(nchan, nbin)
    chirp = torch.roll(chirp, nbin // 2, -1)
    power = torch.zeros((nfft, nchan, nbin), dtype=torch.float64, device=dev)
    for q in range(pol):
        v = torch.fft.ifft((spec[q] * chirp).reshape(nfft, nchan, sft, mbin)) * mbin
        power += (v.real ** 2 + v.imag ** 2).reshape(nfft, nchan, nbin) / nbin / nbin
    del chirp, ang, phase, v
    ovc = nov // sft
    adj = mbin - 2 * ovc
    power = torch.roll(power, nbin // 2, -1).reshape(nfft, nchan, sft, mbin)[..., ovc: ovc + adj]
    plane = power.flip(1, 2).permute(1, 2, 0, 3).reshape(nchan * sft, nfft * adj).contiguous()
    rows, msamp = plane.shape
    foff = (float(fmax) - float(fmin)) / rows
    tw = float(_f32(_f32(sft) * _f32(TSAMP)))
    for i in range(rows):
        f = (rows - 1 - i) * foff + float(fmin)
        d = 4.148808e3 * dm * (1.0 / (float(fmin) * float(fmin)) - 1.0 / (f * f)) / tw
        plane[i] = torch.roll(plane[i], int(math.floor(abs(d) + 0.5) * (1 if d >= 0 else -1)))
    m = plane.mean(1)
    var = plane.var(1, unbiased=False)
    mean = m.mean()
    std = torch.sqrt((var + m * m).mean() - mean * mean)
    bad = (var - var.mean()).abs() > 4.0 * var.std(unbiased=False)
    plane = (plane - mean) / std
    plane[bad] = 0.0
    r0, levels = _keith_plan(fmin, fmax, rows, case["max_dt"])
    mask = (~bad).double()[:, None].expand(rows, msamp).contiguous()
    out = _fdmt64(plane, r0, levels) / torch.sqrt(_fdmt64(mask, r0, levels) + 1e-8)
    return {"planes": out[None], "spectra": torch.view_as_real(spec).reshape(-1, 2)}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("heap", "beams"):   # whole numbers only
        return None
    if kind == "search":
        p = _plane(case["rows"], case["cols"], seed).double()
        return {"stats": torch.cat([p.mean(1), p.std(1, unbiased=False)])}
    if kind == "chunk":
        return _chunk64(case, _raw(case, seed))
    n, d = case["nchan"], case["max_dt"]
    if kind == "adjoint":
        g = torch.Generator(device=_device()).manual_seed(int(seed))
        gy = torch.randn((d, case["ncols"]), generator=g, device=_device())
        return _fdmt64_adjoint(gy.double(), n, *_keith_plan(FMIN, FMAX, n, d))
    x, pulses = _filterbank(n, case["ncols"], d, seed, count=8 if kind == "step" else 3)
    if kind == "pravir":
        return _pravir64(x.double(), d)
    r0, levels = _keith_plan(FMIN, FMAX, n, d)
    x = x.double()
    plane = _fdmt64(x, r0, levels)
    if kind == "fdmt":
        return plane
    y = plane.clone().requires_grad_()
    snr = []
    for row, t0, width in _cells(case, pulses):
        r = y[row]
        z = (r - r.mean()) / r.std(unbiased=False)
        snr.append(z[t0: t0 + width].sum() / math.sqrt(width))
    snr = torch.stack(snr)
    (gy,) = torch.autograd.grad(-snr.sum(), y)
    gx = _fdmt64_adjoint(gy, n, r0, levels)
    return {"plane": plane, "snr": snr.detach(), "grad": (gx * x).sum(1)}
