"""Clustering at the edges of its sizes, against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

from cpp_projects_b200 import cluster, search
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 4864, 4865, 30000])
@pytest.mark.parametrize("metrics", [(0, 0, 0), (-1, 0, 0)])   # by gaps; the sorting passes
def test_groups_at_one_start(cuda, n, metrics):
    """Delegates ordered by a start they all share (a one-column plane, an impulse
    over all rows): nothing to sort by, and more groups than one tile of the sort."""
    c = np.zeros(n, pyoracle.CAND_DTYPE)
    c["mt"] = 17
    c["mdt"] = 3 * np.arange(n)
    c["msnr"] = 7.0 + (np.arange(n) % 5)
    perm, offs, dl = pyoracle.cluster(c, metrics)
    cl = cluster.complete_clusterization(search.cands_from_numpy(c, cuda), metrics)
    np.testing.assert_array_equal(cl.offsets.cpu().numpy(), offs)
    np.testing.assert_array_equal(cl.perm.cpu().numpy(), perm)
    np.testing.assert_array_equal(cl.delegates.cpu().numpy(), dl)


def _pool_high(reset):
    """Most bytes in use of the device's default memory pool (reset: from now on)."""
    rt, pool, v = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p(), ctypes.c_uint64(0)
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    if reset:
        assert rt.cudaMemPoolSetAttribute(pool, 8, ctypes.byref(v)) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 8, ctypes.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("tmax,dmax,metrics", [
    (1 << 26, 1 << 26, (1000, 1000, 1 << 30)),    # two passes of many words, few groups
    (1 << 26, 1 << 29, (1000, 10000, 1 << 30)),   # its first pass by gaps, then too many words
    (4000, 200, (2, 1, 2)), (1 << 26, 64, (64, 1, 1)),
])
def test_scratch_is_bounded(cuda, tmax, dmax, metrics):
    """48 bytes per candidate, and per group its 64 delegate lanes and four words."""
    n = 3 << 20
    g = torch.Generator(device=cuda).manual_seed(tmax)
    f = [torch.randint(0, m, (n,), generator=g, device=cuda) for m in (tmax, dmax, 6, 1 << 20)]
    c = torch.stack(f, 1).to(torch.int32)
    cluster.complete_clusterization(c, metrics)
    torch.cuda.synchronize()
    before = _pool_high(True)
    cl = cluster.complete_clusterization(c, metrics)
    used, groups = _pool_high(False) - before, cl.offsets.shape[0] - 1
    assert used <= 48 * n + (64 * 8 + 16) * groups + (8 << 20), (used / n, groups)
