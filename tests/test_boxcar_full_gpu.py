"""Thresholds near the noise search the plane unfiltered (k_boxcar_full): both
sides of every line of that rule against the oracle's exhaustive search, for
thresholds on the host and in device memory."""
import ctypes

import numpy as np
import pytest
import torch

from cpp_projects_b200 import _capi, search
from cpp_projects_b200._tensors import dev_ptr, stream_handle
from oracle import pyoracle

pytestmark = pytest.mark.gpu

CAP = 1 << 22


def _gather(plane, stats, thr, mode, param, on_device, cuda):
    rows, cols = plane.shape
    out, n = torch.zeros((CAP, 4), dtype=torch.int32, device=cuda), ctypes.c_uint32(0)
    t = torch.tensor([thr], device=cuda)
    _capi.call("bfs_boxcar_gather", dev_ptr(plane), rows, cols, None if stats is None else dev_ptr(stats),
               ctypes.c_float(-1e9 if on_device else thr), dev_ptr(t) if on_device else None, mode, param, 0, dev_ptr(out),
               ctypes.c_uint32(CAP), ctypes.byref(n), stream_handle())
    return search.cands_to_numpy(out[: n.value])


@pytest.mark.parametrize("mode,param", [(0, 0), (0, 2), (0, 5), (0, 7), (1, 1), (1, 3), (1, 8)])
# 64 x 16000: 32 row pairs x 63 tiles, just over the rule's fewest; 63 x 16129: an odd row, ragged and unaligned
# rows; 61 x 16128: one tile short of it
@pytest.mark.parametrize("rows,cols,off", [(64, 16000, 0), (63, 16129, 1), (61, 16128, 0)])
def test_low_thresholds(cuda, mode, param, rows, cols, off):
    rng = np.random.default_rng(rows + param)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    x[1, 100:140] += 3.0
    x[2, cols - 1] = 9.0
    x[3, 5000] = np.nan
    x[4, 255] = np.inf
    x[rows - 1, :8] = 6.0
    m, sd = rng.uniform(-2, 2, rows).astype(np.float32), rng.uniform(0.5, 3, rows).astype(np.float32)
    sd[5] = 0.0
    raw = torch.empty(rows * cols + off, device=cuda)[off:].view(rows, cols)   # 4 bytes off a 16-byte boundary
    with np.errstate(all="ignore"):
        raw.copy_(torch.from_numpy((x * np.where(sd > 0, sd, 1)[:, None] + m[:, None]).astype(np.float32)))
        r = raw.cpu().numpy()
        z = np.where(sd[:, None] > 0, ((r - m[:, None]).astype(np.float32) / sd[:, None]).astype(np.float32), np.float32(0))
    stats = torch.from_numpy(np.concatenate([m, sd])).to(cuda)
    for thr in (0.9, 1.1, 3.0, 4.0, 4.7, 5.1, 5.9, 7.0):
        want = pyoracle.boxcar(z.astype(np.float32), thr, mode, param)
        if len(want) > CAP:
            continue
        for on_device in (False, True):
            got = _gather(raw, stats, thr, mode, param, on_device, cuda)
            assert len(got) == len(want), (thr, on_device)
            for k in ("mt", "mdt", "mwidth", "msnr"):
                np.testing.assert_array_equal(got[k].view(np.uint32), want[k].view(np.uint32))


def test_overflow_at_a_low_threshold(cuda):
    """More candidates than room, found unfiltered from a device threshold: the count, and the error."""
    x = torch.randn((64, 16000), generator=torch.Generator(device=cuda).manual_seed(2), device=cuda)
    want = len(pyoracle.boxcar(x.cpu().numpy(), 3.0, 0, 5))
    t, out, n = torch.tensor([3.0], device=cuda), torch.zeros((100, 4), dtype=torch.int32, device=cuda), ctypes.c_uint32(0)
    with pytest.raises(_capi.BfsError, match="OVERFLOW"):
        _capi.call("bfs_boxcar_gather", dev_ptr(x), 64, 16000, None, ctypes.c_float(0.0), dev_ptr(t), 0, 5, 0, dev_ptr(out),
                   ctypes.c_uint32(100), ctypes.byref(n), stream_handle())
    assert n.value == want


def test_batched_search_at_a_low_threshold(cuda):
    from cpp_projects_b200.pipeline import BatchedSearch, BeamShape, SearchPipeline
    shapes = [BeamShape(n, c, 1200.0, 1600.0, n) for n, c in ((64, 16000), (128, 9001), (64, 500))]
    g = torch.Generator(device=cuda).manual_seed(4)
    x = [torch.randn((s.nchan, s.nsamp), generator=g, device=cuda) for s in shapes]
    batch = BatchedSearch(shapes, thr=4.0, capacity=1 << 20)
    plain = SearchPipeline(shapes, thr=4.0, capacity=1 << 20, device=cuda).run(x)
    for _ in range(2):   # eager, then captured
        for a, b in zip(batch.run(x), plain):
            assert a.n_candidates == b.n_candidates > 0
            np.testing.assert_array_equal(a.delegates, b.delegates)
            np.testing.assert_array_equal(a.group_sizes, b.group_sizes)
