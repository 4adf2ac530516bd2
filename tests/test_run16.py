"""Run segments over 16-bit planes (k_fdmt_run16).  CPU: every tile replayed as
the kernel indexes shared memory (16-byte copies, kept inputs, words cut at odd
offsets), on whole numbers that need no rounding, against the level planes;
shared memory starts as NaN, so a written sample that depended on a value never
loaded would differ.  GPU: bit for bit the plain passes (seg_levels = 1), which
other tests hold to the oracle, over ragged lengths, odd output rows, values
whose sums leave the 16-bit range, infinities and NaN."""
import ctypes

import numpy as np
import pytest
import torch

from cpp_projects_b200 import CFdmtGpu, _capi
from oracle import pyoracle
from test_seg_plan import level_planes, merge_level

P = ctypes.c_void_p
TT, MID, WARPS = 512, 576, 8


def plan16(nchan, ncols, max_dt, fuse=-1):
    desc = _capi.FdmtDesc(fmin=1200.0, fmax=1600.0, nchan=nchan, ncols=ncols, max_dt=max_dt, fuse_depth=fuse, precision=1)
    plan = P()
    _capi.call("bfs_fdmt_plan_create_host", ctypes.byref(desc), ctypes.byref(plan))
    try:
        n = ctypes.c_int(0)
        _capi.call("bfs_fdmt_plan_passes", plan, ctypes.byref(n), None, 0)
        pp = np.zeros(13 * n.value, np.int32)
        _capi.call("bfs_fdmt_plan_passes", plan, ctypes.byref(n), pp.ctypes.data_as(P), pp.size)
        out = []
        for i in range(n.value):
            pr = np.zeros(14, np.int32)
            _capi.call("bfs_fdmt_plan_run", plan, i, pr.ctypes.data_as(P), None, 0, None, 0, None, 0)
            t, r, e = (np.zeros(k, np.int32) for k in (8 * pr[11], 2 * pr[12], 4 * pr[13]))
            if pr[0]:
                _capi.call("bfs_fdmt_plan_run", plan, i, pr.ctypes.data_as(P), t.ctypes.data_as(P), t.size,
                           r.ctypes.data_as(P), r.size, e.ctypes.data_as(P), e.size)
            out.append((int(pp[13 * i]), int(pp[13 * i + 1]), pr, t.reshape(-1, 8), r.reshape(-1, 2), e.reshape(-1, 4)))
        return out
    finally:
        _capi.lib().bfs_fdmt_plan_destroy(plan)


def emulate(src, pr, tiles, rows, ent, ncols, out_rows):
    s1, s2, r0c, pitch, zx, y0, zy, ent0, max_ent, _ = (int(v) for v in pr[:10])
    assert r0c == 0 and pitch % 8 == 0 and ent0 % 8 == 0 and int(pr[10]) == 2 * ent0 + 32 * max_ent <= 113 * 1024
    out = np.full((out_rows, ncols), np.nan)
    for row0, e0, n_in, n1, n2, out0, _, _ in tiles:
        assert n_in <= 32 * WARPS and n_in * pitch <= zx and y0 + n1 * MID <= zy and n1 + n2 < max_ent
        for t0 in range(0, ncols, TT):
            sm = np.full(ent0, np.nan)
            sm[zx:zx + MID] = 0.0
            sm[zy:zy + TT] = 0.0
            for j, (row, lead) in enumerate(rows[row0:row0 + n_in]):
                assert lead % 8 == 0
                t = t0 - lead + np.arange(pitch)
                sm[j * pitch:(j + 1) * pitch] = np.where((t >= 0) & (t < ncols), src[row][np.clip(t, 0, ncols - 1)], 0.0)

            def stage(e, n, levels, cols, put):
                for w in range(WARPS):
                    kept = [None] * 4
                    for r in range(n * w // WARPS, n * (w + 1) // WARPS):
                        for i in range(2 * levels):
                            q = int(e[r][i])
                            if q & 1 or kept[i] is None:
                                off = (q & ~1) // 2
                                # the words read: from the even offset below, one more for an odd one
                                assert 0 <= off - (off & 1) and off + cols + (off & 1) <= ent0
                                kept[i] = sm[off:off + cols].copy()
                        v = kept[0] + kept[1]
                        put(r, v + (kept[2] + kept[3]) if levels == 2 else v)

            stage(ent[e0:e0 + n1], n1, s1, MID, lambda r, v: sm.__setitem__(slice(y0 + r * MID, y0 + (r + 1) * MID), v))

            def store(r, v):
                n = min(TT, ncols - t0)
                out[out0 + r, t0:t0 + n] = v[:n]

            stage(ent[e0 + n1:e0 + n1 + n2], n2, s2, TT, store)
    return out


@pytest.mark.parametrize("nchan,ncols,max_dt", [(64, 1300, 64), (256, 1025, 256), (128, 511, 200), (512, 1537, 300)])
def test_run16_plan_replayed(nchan, ncols, max_dt):
    x = np.random.default_rng(3).integers(-8, 9, size=(nchan, ncols)).astype(np.float32)
    passes = plan16(nchan, ncols, max_dt)
    planes = level_planes(1200.0, 1600.0, x, nchan, ncols, max_dt, passes[-1][1])
    assert passes[0][2][0] > 0 and 1 << passes[-1][1] == nchan
    rng = np.random.default_rng(4)
    for l0, l1, pr, tiles, rows, ent in passes:
        src = rng.integers(-50, 51, size=planes[l0].shape).astype(np.float32)   # sums of whole numbers: exact
        want = src
        for level in range(l0 + 1, l1 + 1):
            want = merge_level(want, *pyoracle.fdmt_tables(1200.0, 1600.0, nchan, max_dt, level))
        got = emulate(src, pr, tiles, rows, ent, ncols, planes[l1].shape[0])
        assert np.array_equal(got, want)


def test_run16_needs_equal_scales():
    # rows of a level that sum different numbers of channels: plain passes
    assert all(p[2][0] == 0 for p in plan16(100, 2048, 77))
    # an explicit depth 0 and one level per pass stay plain
    assert all(p[2][0] == 0 for p in plan16(64, 1000, 64, fuse=0))


def _same(a, b):
    a, b = a.view(torch.int32), b.view(torch.int32)
    an, bn = torch.isnan(a.view(torch.float32)), torch.isnan(b.view(torch.float32))
    return bool(torch.equal(an, bn) and torch.equal(a[~an], b[~bn]))


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("nchan,ncols,max_dt", [(8, 40, 8), (64, 511, 64), (64, 1000, 100), (128, 513, 40), (256, 1, 256),
                                                (1024, 3001, 1024), (4096, 2050, 4096)])
@pytest.mark.parametrize("kind", ["noise", "tiny", "large", "special"])
def test_run16_equals_plain_passes(cuda, prec, nchan, ncols, max_dt, kind):
    g = torch.Generator(device=cuda).manual_seed(nchan + ncols)
    x = torch.randn((nchan, ncols), generator=g, device=cuda)
    if kind == "tiny":      # 16-bit subnormals and sums on their border
        x = x * (2.0 ** -17 if prec == 1 else 2.0 ** -129)
    elif kind == "large":   # stored values near the top of the range: their sums pass it
        x = torch.sign(x) * (40000.0 + 1000.0 * x) if prec == 1 else x * 1e36
    elif kind == "special":
        x[::5, ::97] = float("inf")
        x[1::7, ::89] = -float("inf")
        x[2::11, ::101] = float("nan")
        x[3::4] = -0.0
    plans = [CFdmtGpu(1200.0, 1600.0, nchan, ncols, max_dt, fuse_depth=2, precision=prec, seg_levels=s) for s in (0, 1)]
    assert plans[0].info.hbm_passes < plans[1].info.hbm_passes or nchan < 16
    out = torch.full((2, max_dt, ncols + 1), 7.0, device=cuda)
    flat = [torch.full((max_dt * ncols + 1,), 7.0, device=cuda)[1:] for _ in plans]   # off the 8-byte boundary
    for f, o in zip(plans, flat):
        f.process_image(x, o.view(max_dt, ncols), False)
        f.process_image(x, out[0].view(-1)[:max_dt * ncols].view(max_dt, ncols), False)
        assert _same(o, out[0].view(-1)[:max_dt * ncols].reshape(-1))
    assert _same(flat[0], flat[1])
