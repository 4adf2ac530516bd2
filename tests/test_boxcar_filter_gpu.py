"""The boxcar's tile filter drops no window: planes whose windows sit just
above and just below the threshold in noise-free tiles, at every edge of the
filter's blocks, against the oracle's exhaustive search."""
import numpy as np
import pytest
import torch

from cpp_projects_b200 import search
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _same(plane, mode, param, thr, stats, cuda):
    z = plane
    if stats is not None:
        r = plane.shape[0]
        with np.errstate(all="ignore"):
            d = (plane - stats[:r, None]).astype(np.float32)
            z = np.where(stats[r:, None] > 0, (d / stats[r:, None]).astype(np.float32), np.float32(0))
    want = pyoracle.boxcar(z.astype(np.float32), thr, mode, param)
    st = None if stats is None else torch.from_numpy(stats).to(cuda)
    got, n = search.boxcar_gather(torch.from_numpy(plane).to(cuda), thr, mode, param, stats=st, capacity=1 << 20)
    got = search.cands_to_numpy(got)
    assert n == len(want)
    for k in ("mt", "mdt", "mwidth", "msnr"):
        np.testing.assert_array_equal(got[k].view(np.uint32), want[k].view(np.uint32))
    return n


@pytest.mark.parametrize("mode,param", [(0, q) for q in range(8)] + [(1, w) for w in range(1, 9)])
@pytest.mark.parametrize("cols", [600, 1031])
def test_windows_at_the_threshold_are_found(cuda, mode, param, cols):
    thr = 7.0
    widths = [1 << k for k in range(param + 1)] if mode == 0 else range(1, param + 1)
    rows = []
    for w in widths:
        for start in (0, 3, 7, 8, 200, 249, 255, 256 - w // 2, 300, cols - w):
            for scale in (0.99998, 1.0, 1.00002):   # one flat window of S/N thr * scale
                x = np.zeros(cols, np.float32)
                x[max(0, start):start + w] = np.float32(thr * scale / np.sqrt(w))
                rows.append(x)
    plane = np.stack(rows)
    n = _same(plane, mode, param, thr, None, cuda)
    assert n > 0
    # the same planes away from mean 0 and deviation 1 (statistics given, not computed)
    rng = np.random.default_rng(param)
    m = rng.uniform(-3, 3, len(rows)).astype(np.float32)
    sd = rng.uniform(0.3, 40, len(rows)).astype(np.float32)
    raw = (plane * sd[:, None] + m[:, None]).astype(np.float32)
    _same(raw, mode, param, thr, np.concatenate([m, sd]), cuda)


@pytest.mark.parametrize("thr", [3.0, 0.5, 0.0, -1.0])
def test_low_and_negative_thresholds_and_special_values(cuda, thr):
    rng = np.random.default_rng(5)
    x = rng.standard_normal((9, 700)).astype(np.float32)
    x[1, 100] = np.nan
    x[2, 260] = np.inf
    x[3, 10] = -np.inf
    x[4, 500] = 3e38
    x[4, 505] = 3e38
    x[5] = 0
    stats = np.concatenate([np.zeros(9), np.ones(9)]).astype(np.float32)
    stats[9 + 5] = 0.0         # a constant row
    stats[9 + 6] = 1e-40       # deviations outside the filter's range
    stats[9 + 7] = 1e36
    for mode, param in ((0, 5), (1, 4)):
        _same(x, mode, param, thr, None, cuda)
        _same(x, mode, param, thr, stats, cuda)
