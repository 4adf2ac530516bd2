"""CPU: adjoint run segments (k_adj_run) replayed from their tiles and blobs
against the level-by-level adjoint, bit for bit; shared memory starts as NaN.
GPU: the same shapes through the library against the oracle."""
import ctypes

import numpy as np
import pytest

from cpp_projects_b200 import _capi
from oracle import pyoracle

P = ctypes.c_void_p
TT, MID = 256, 288


def adjoint_runs(nchan, ncols, max_dt):
    desc = _capi.FdmtDesc(fmin=1200.0, fmax=1600.0, nchan=nchan, ncols=ncols, max_dt=max_dt, fuse_depth=0,
                          seg_levels=1)
    plan = ctypes.c_void_p()
    _capi.call("bfs_fdmt_plan_create_host", ctypes.byref(desc), ctypes.byref(plan))
    try:
        out, i = [], 0
        while True:
            pr = np.zeros(12, np.int32)
            _capi.call("bfs_fdmt_plan_adjoint_run", plan, i, pr.ctypes.data_as(P), None, 0, None, 0, None, 0)
            if i >= pr[0]:
                return out
            t, r, b = (np.zeros(k, np.int32) for k in (8 * pr[9], 2 * pr[10], pr[11]))
            _capi.call("bfs_fdmt_plan_adjoint_run", plan, i, pr.ctypes.data_as(P), t.ctypes.data_as(P), t.size,
                       r.ctypes.data_as(P), r.size, b.ctypes.data_as(P), b.size)
            out.append((pr, t.reshape(-1, 8), r.reshape(-1, 2), b))
            i += 1
    finally:
        _capi.lib().bfs_fdmt_plan_destroy(plan)


def emulate(src, pr, tiles, rows, blob, ncols, nout):
    _, l0, l1, final, pitch, y0, blob0, max_blob, max_e = (int(v) for v in pr[:9])
    f32 = np.float32
    out = np.full((nout, ncols), np.nan, np.float32)
    written = np.zeros((nout, ncols), np.int32)
    for row0, b0, n, n_in, n1, n2, e_max, _ in tiles:
        assert n % 4 == 0 and n <= max_blob and n_in * pitch <= y0 - MID and y0 + n1 * MID <= blob0 - TT
        B = blob[b0:b0 + n].astype(np.int64)
        H = B[n1:]
        for t0 in range(0, ncols + int(e_max), TT):
            sm = np.full(blob0, np.nan, np.float32)
            for j, (row, lead) in enumerate(rows[row0:row0 + n_in]):
                t = t0 - lead + np.arange(pitch)
                v = np.zeros(pitch, np.float32)
                ok = (t >= 0) & (t < ncols)
                v[ok] = src[row, t[ok]]
                sm[j * pitch:(j + 1) * pitch] = v

            def load(q, cols, lo, hi):
                off = int(q & 0xffffc) >> 2
                assert lo <= off and off + cols <= hi
                return sm[off:off + cols]

            def terms(at):
                k = int(at) & ~3
                kind, got = int(at) & 3, []
                while kind != 3 and not (got and got[-1] & (1 << 28)):
                    got.append(int(B[k]))
                    k += 1
                assert kind != 1 or [q & 1 for q in got] == [0, 1, 0, 1]
                assert kind != 2 or [q & 1 for q in got] == [1, 1]
                return got

            for r in range(n1):
                acc = np.zeros(MID, np.float32)
                part = np.zeros(MID, np.float32)
                for q in terms(B[r]):
                    part = part + load(q, MID, 0, y0)
                    if q & 1:
                        acc, part = acc + part, np.zeros(MID, np.float32)
                sm[y0 + r * MID:y0 + (r + 1) * MID] = acc
            for r in range(n2):
                row, u = int(H[3 * r]), t0 - int(H[3 * r + 1]) + np.arange(TT)
                part, g, w, gx = (np.zeros(TT, np.float32) for _ in range(4))
                for q in terms(H[3 * r + 2]):
                    part = part + load(q, TT, y0, blob0)
                    if q & 1:
                        g, part = g + part, np.zeros(TT, np.float32)
                    if final and q & 2:
                        rr, k = (q >> 20) & 7, (q >> 23) & 7
                        w = np.where(u + k >= rr, w + g, w)
                        g = np.zeros(TT, np.float32)
                        if q & (1 << 26):
                            gx, w = gx + w * (f32(1) / f32(rr + 1)), np.zeros(TT, np.float32)
                ok = (u >= 0) & (u < ncols)
                out[row, u[ok]] = (gx if final else g)[ok]
                written[row, u[ok]] += 1
    assert np.all(written == 1)
    return out


def adjoint_level(gout, a, b, s, nin):
    ncols = gout.shape[1]
    gin = np.zeros((nin, ncols), np.float32)
    for g in range(len(a)):
        gin[a[g]] += gout[g]
        if b[g] >= 0 and s[g] < ncols:
            gin[b[g], :ncols - s[g]] += gout[g, s[g]:]
    return gin


CASES = [(64, 700, 64), (64, 1024, 64), (96, 601, 96), (100, 900, 150), (128, 777, 64), (64, 530, 200),
         (33, 400, 40), (5, 300, 9), (256, 515, 256), (8, 64, 8)]


@pytest.mark.parametrize("case", CASES)
def test_adjoint_runs_replayed_match_the_levels(case):
    nchan, ncols, max_dt = case
    segs = adjoint_runs(nchan, ncols, max_dt)
    nrows = pyoracle.fdmt_rows(1200.0, 1600.0, nchan, max_dt)
    assert segs and segs[0][0][2] == len(nrows) - 1
    assert segs[-1][0][3] == (nrows[0] // nchan <= 5)   # more level-0 rows: their plane, then the running-mean adjoint
    gy = np.random.default_rng(nchan + ncols).standard_normal((max_dt, ncols)).astype(np.float32)
    gy[:, ::7] = np.float32(-0.0)
    g = gy
    for pr, tiles, rows, blob in segs:
        l0, l1, final = (int(v) for v in pr[1:4])
        got = emulate(g, pr, tiles, rows, blob, ncols, nchan if final else int(nrows[l0]))
        want = g
        for lev in range(l1, l0, -1):
            a, b, s = pyoracle.fdmt_tables(1200.0, 1600.0, nchan, max_dt, lev)
            want = adjoint_level(want, a, b, s, int(nrows[lev - 1]))
        if final:
            want = pyoracle.fdmt_adjoint_f32(1200.0, 1600.0, gy, nchan, ncols, max_dt)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), f"levels {l1}..{l0}"
        g = got


@pytest.mark.parametrize("nchan,max_dt", [(256, 256), (512, 512), (1024, 1024), (4096, 4096), (512, 768)])
def test_search_shapes_have_adjoint_runs(nchan, max_dt):
    segs = adjoint_runs(nchan, 20001, max_dt)
    assert segs and all(4 * (int(p[6]) + 2 * int(p[7])) <= 113 * 1024 for p, _, _, _ in segs)


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES + [(1024, 4099, 1024), (512, 20000, 512), (256, 60001, 256)])
@pytest.mark.parametrize("shift", [0, 1])   # gradient base on and off a 16-byte boundary
def test_adjoint_runs_bit_exact_vs_oracle(cuda, case, shift):
    import torch
    from cpp_projects_b200 import CFdmtGpu
    nchan, ncols, max_dt = case
    gy = np.random.default_rng(nchan + ncols).standard_normal((max_dt, ncols)).astype(np.float32)
    gy[:, ::7] = np.float32(-0.0)
    buf = torch.zeros(gy.size + 4, device=cuda)
    d = buf[shift:shift + gy.size].view(max_dt, ncols)
    d.copy_(torch.from_numpy(gy))
    gx = CFdmtGpu(1200.0, 1600.0, nchan, ncols, max_dt).adjoint(d).cpu().numpy()
    want = pyoracle.fdmt_adjoint_f32(1200.0, 1600.0, gy, nchan, ncols, max_dt)
    assert np.array_equal(gx.view(np.uint32), want.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,shift", [(5, 8192, 0), (3, 8193, 0), (4, 40004, 1), (2, 3, 0), (3, 100, 0)])
def test_snr_gradient_parts_match_fp64(cuda, rows, cols, shift):
    """Row parts, 16-byte groups and their ends: one cell at each edge of a part."""
    import torch
    from cpp_projects_b200 import search
    g = torch.Generator().manual_seed(rows * cols)
    buf = torch.zeros(rows * cols + 4, device=cuda)
    y = buf[shift:shift + rows * cols].view(rows, cols)
    y.copy_(torch.randn(rows, cols, generator=g))
    spans = [(0, 1), (max(0, cols - 3), min(3, cols)), (min(8190, cols - 1), min(4, cols - min(8190, cols - 1)))]
    cells = [[r, t, w] for r in range(rows - 1) for t, w in spans]   # the last row has none
    st = search.row_stats(y)
    snr = search.snr_cells(y, st, cells)
    gs = torch.randn(len(cells), generator=g).to(cuda)
    got = search.snr_cells_adjoint(y, st, cells, snr, gs)
    y64 = y.double().cpu().requires_grad_()
    m, sd = y64.mean(1), y64.std(1, unbiased=False)
    s = torch.stack([((y64[r, t:t + w] - m[r]) / sd[r]).sum() / w ** 0.5 for r, t, w in cells])
    (want,) = torch.autograd.grad((s * gs.double().cpu()).sum(), y64)
    # statistics and S/N are rounded to float (2^-24 each) and a few products of them summed
    scale = want.abs().max().item() + 1e-30
    assert (got.double().cpu() - want).abs().max().item() < 32 * 2.0 ** -24 * scale * max(1.0, snr.abs().max().item())
    assert torch.all(got[-1] == 0)
