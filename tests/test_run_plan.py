"""CPU: run segments (k_fdmt_run) replayed as the kernel indexes shared memory
-- every copy, kept register, merge and store of every tile -- against the
level planes, bit for bit.  Shared memory starts as NaN, so a written sample
that depended on a value never loaded would differ.  GPU: the same shapes
through the library against the oracle."""
import ctypes

import numpy as np
import pytest

from cpp_projects_b200 import _capi
from oracle import pyoracle
from test_seg_plan import level_planes, merge_level

P = ctypes.c_void_p
TT, MID, WARPS = 256, 288, 8


def plan_runs(fmin, fmax, nchan, ncols, max_dt, fuse, seg_levels):
    """[(l0, l1, params, tiles, rows, ent)] of a plan's passes and its level rows."""
    desc = _capi.FdmtDesc(fmin=fmin, fmax=fmax, nchan=nchan, ncols=ncols, max_dt=max_dt, fuse_depth=fuse,
                          seg_levels=seg_levels)
    plan = ctypes.c_void_p()
    _capi.call("bfs_fdmt_plan_create_host", ctypes.byref(desc), ctypes.byref(plan))
    try:
        info = _capi.FdmtInfo()
        _capi.call("bfs_fdmt_plan_info", plan, ctypes.byref(info))
        rows = np.zeros(info.niter + 1, np.int32)
        _capi.call("bfs_fdmt_plan_rows", plan, rows.ctypes.data_as(P), rows.size)
        n = ctypes.c_int(0)
        _capi.call("bfs_fdmt_plan_passes", plan, ctypes.byref(n), None, 0)
        pp = np.zeros(13 * n.value, np.int32)
        _capi.call("bfs_fdmt_plan_passes", plan, ctypes.byref(n), pp.ctypes.data_as(P), pp.size)
        out = []
        for i in range(n.value):
            pr = np.zeros(14, np.int32)
            _capi.call("bfs_fdmt_plan_run", plan, i, pr.ctypes.data_as(P), None, 0, None, 0, None, 0)
            t, r, e = (np.zeros(k, np.int32) for k in (8 * pr[11], 2 * pr[12], 4 * pr[13]))
            _capi.call("bfs_fdmt_plan_run", plan, i, pr.ctypes.data_as(P), t.ctypes.data_as(P), t.size,
                       r.ctypes.data_as(P), r.size, e.ctypes.data_as(P), e.size)
            out.append((int(pp[13 * i]), int(pp[13 * i + 1]), pr, t.reshape(-1, 8), r.reshape(-1, 2),
                        e.reshape(-1, 4)))
        return int(info.fuse_depth), rows, out
    finally:
        _capi.lib().bfs_fdmt_plan_destroy(plan)


def emulate_run(src, pr, tiles, rows, ent, ncols, out_rows):
    s1, s2, r0c, pitch, zx, y0, zy, ent0, max_ent, edge = (int(v) for v in pr[:10])
    assert pitch % 4 == 0 and ent0 % 4 == 0 and int(pr[10]) == 4 * ent0 + 32 * max_ent
    out = np.full((out_rows, ncols), np.nan, np.float32)
    written = np.zeros(out_rows, np.int64)
    f32 = np.float32
    for row0, e0, n_in, n1, n2, out0, _, _ in tiles:
        assert n_in <= 32 * WARPS and n_in * pitch <= zx and y0 + n1 * MID <= zy and n1 + n2 <= max_ent
        for t0 in range(0, ncols, TT):
            sm = np.full(ent0, np.nan, np.float32)
            sm[zx:zx + MID] = f32(-0.0)
            sm[zy:zy + TT] = f32(-0.0)
            for j, (row, lead) in enumerate(rows[row0:row0 + n_in]):
                assert ((row * ncols if r0c else 0) + t0 - lead) % 4 == 0
                t = t0 - lead + np.arange(pitch)
                v = np.where(t < 0, f32(-0.0), f32(0.0))
                ok = (t >= 0) & (t < ncols)
                v[ok] = src[row, t[ok]]
                sm[j * pitch:(j + 1) * pitch] = v

            def read(q, cols, lo, hi, chan):
                off, r = (q & 0xffffc) >> 2, q >> 20
                idx = off + np.arange(cols)
                assert idx.min() - r >= lo and idx.max() < hi
                v = sm[idx].copy()
                for k in range(1, r + 1):
                    m = v if k == 1 else (v * f32(k)).astype(np.float32)
                    v = ((m + sm[idx - k]).astype(np.float32) / f32(k + 1)).astype(np.float32)
                if r:
                    assert chan and r < r0c
                    j = off // pitch
                    t = t0 - rows[row0 + j][1] + off - j * pitch + np.arange(cols)
                    if t0 < edge:
                        v = np.where(t < 0, f32(-0.0), np.where(t < r, f32(0.0), v))
                    # (elsewhere no column that is used precedes sample r)
                return v

            def stage(e, n, levels, cols, lo, hi, put, chan=False):
                for w in range(WARPS):
                    a, b = n * w // WARPS, n * (w + 1) // WARPS
                    v = [None] * 4
                    for r in range(a, b):
                        for i in range(2 * levels):
                            q = int(e[r][i]) | (1 if r == a else 0)
                            if q & 1:
                                v[i] = read(q & ~1, cols, lo, hi, chan)
                        o = (v[0] + v[1]).astype(np.float32)
                        if levels == 2:
                            o = (o + (v[2] + v[3]).astype(np.float32)).astype(np.float32)
                        put(r, o)

            def put_mid(r, o):
                sm[y0 + r * MID:y0 + (r + 1) * MID] = o

            def put_out(r, o):
                n = min(TT, ncols - t0)
                out[out0 + r, t0:t0 + n] = o[:n]
                written[out0 + r] += n

            stage(ent[e0:e0 + n1], n1, s1, MID, 0, y0, put_mid, chan=r0c > 0)
            stage(ent[e0 + n1:e0 + n1 + n2], n2, s2, TT, y0, ent0, put_out)
    assert np.all(written == ncols)
    return out


CASES = [  # nchan, ncols, max_dt, seg_levels: odd lengths, odd sub-band counts, 2-5 level-0 rows
    (64, 700, 64, 3), (64, 1024, 64, 4), (64, 515, 64, 2), (96, 601, 96, 4), (100, 900, 150, 3),
    (128, 777, 64, 4), (64, 530, 200, 3), (33, 400, 40, 2), (5, 300, 9, 3), (256, 258, 256, 4),
]


@pytest.mark.parametrize("case", CASES)
def test_run_segments_replayed_match_the_level_planes(case):
    nchan, ncols, max_dt, levels = case
    k, nrows, passes = plan_runs(1200.0, 1600.0, nchan, ncols, max_dt, 0, levels)
    assert k == 0 and any(p[2][0] for p in passes)
    x = np.random.default_rng(nchan + ncols).standard_normal((nchan, ncols)).astype(np.float32)
    x[:, ::7] = np.float32(-0.0)
    x[::3, 5::11] = np.float32(1e-40)
    planes = level_planes(1200.0, 1600.0, x, nchan, ncols, max_dt, nrows.size - 1)
    for l0, l1, pr, tiles, rows, ent in passes:
        if pr[0] == 0:
            continue
        got = emulate_run(x if pr[2] else planes[l0], pr, tiles, rows, ent, ncols, int(nrows[l1]))
        assert np.array_equal(got.view(np.uint32), planes[l1].view(np.uint32)), f"levels {l0}..{l1}"


@pytest.mark.parametrize("nchan", [256, 512, 1024, 4096])
@pytest.mark.parametrize("levels", [2, 3, 4])
def test_search_shapes_run_in_two_ctas_per_sm(nchan, levels):
    _, _, passes = plan_runs(1200.0, 1600.0, nchan, 30001, nchan, 0, levels)
    for l0, l1, pr, tiles, rows, ent in passes:
        if l1 - l0 < 2:
            continue
        assert pr[0] + pr[1] == l1 - l0 and pr[10] <= 113 * 1024
        bytes_ = ent & 0xffffc
        assert bytes_.max() + 4 * MID <= 4 * (pr[7] + MID) and pr[3] <= 384


@pytest.mark.gpu
@pytest.mark.parametrize("case", [(64, 1000, 64, 1, 0), (96, 701, 96, 1, 0), (33, 515, 100, 1, 0), (128, 2050, 50, 1, 0),
                                  (1024, 3001, 1024, 1, 0), (64, 900, 64, 2, 0), (64, 900, 64, 1, 3)])
def test_pravir_plans_bit_exact_vs_oracle(cuda, case):
    """Delays 0, 1, 2, .. per channel form level 0 on chip, other grids in a plane."""
    import torch
    from cpp_projects_b200.fdmt import FDMTGPU
    nchan, ncols, max_dt, step, lo = case
    x = np.random.default_rng(nchan + ncols).standard_normal((nchan, ncols)).astype(np.float32)
    x[:, ::7] = np.float32(-0.0)
    x[::3, 5::11] = np.float32(-1e-40)
    got = FDMTGPU(1200.0, 1600.0, nchan, ncols, 1e-3, max_dt, step, lo)(torch.from_numpy(x).to(cuda)).cpu().numpy()
    want = pyoracle.pravir_fdmt(1200.0, 1600.0, x, nchan, ncols, max_dt, step, lo)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES + [(1024, 4099, 1024, 4), (512, 20000, 512, 3), (256, 60001, 256, 4)])
@pytest.mark.parametrize("shift", [0, 1])   # input base on and off a 16-byte boundary
def test_run_segments_bit_exact_vs_oracle(cuda, case, shift):
    import torch
    from cpp_projects_b200 import CFdmtGpu
    nchan, ncols, max_dt, levels = case
    x = np.random.default_rng(nchan + ncols).standard_normal((nchan, ncols)).astype(np.float32)
    x[:, ::7] = np.float32(-0.0)
    x[::3, 5::11] = np.float32(1e-40)
    buf = torch.zeros(x.size + 4, device=cuda)
    d = buf[shift:shift + x.size].view(nchan, ncols)
    d.copy_(torch.from_numpy(x))
    f = CFdmtGpu(1200.0, 1600.0, nchan, ncols, max_dt, fuse_depth=0, seg_levels=levels)
    got = f(d).cpu().numpy()
    want = pyoracle.fdmt_f32(1200.0, 1600.0, x, nchan, ncols, max_dt)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
