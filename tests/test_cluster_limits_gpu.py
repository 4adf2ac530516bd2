"""Clustering at the edges of its sizes, against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

from cpp_projects_b200 import _capi, cluster, search
from cpp_projects_b200._tensors import dev_ptr, stream_handle
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


@pytest.mark.parametrize("top", [4, 7])   # below ngroups0, and ids that fit its bits but not the count
def test_initial_groups_beyond_the_count(cuda, top):
    """Ids of 0..ngroups0-1 are asked for; larger ones take the sorting passes, which
    have no table of them: the groups are those of each id's candidates alone."""
    rng = np.random.default_rng(top)
    n, ids = 3000, np.sort(rng.integers(0, top + 1, 3000)).astype(np.int32)
    ids[-1] = top
    c = np.zeros(n, pyoracle.CAND_DTYPE)
    c["mt"], c["mdt"], c["mwidth"] = rng.integers(0, 900, n), rng.integers(0, 60, n), rng.integers(0, 6, n)
    c["msnr"] = 7.0 + rng.integers(0, 9, n)
    g0, d = torch.from_numpy(ids).to(cuda), search.cands_from_numpy(c, cuda)
    perm, dl = torch.empty((2, n), dtype=torch.int32, device=cuda)
    offs, ng = torch.empty(n + 1, dtype=torch.int32, device=cuda), ctypes.c_uint32(0)
    metrics = (2, 1, 2)
    _capi.call("bfs_cluster_grouped", dev_ptr(d), ctypes.c_uint32(n), dev_ptr(g0), ctypes.c_uint32(5),
               (ctypes.c_int * 3)(*metrics), dev_ptr(perm), dev_ptr(offs), dev_ptr(dl), ctypes.byref(ng), stream_handle())
    wperm, woffs = [], [0]
    for i in range(top + 1):
        at = np.flatnonzero(ids == i)
        if len(at):
            p, o, _ = pyoracle.cluster(c[at], metrics)
            wperm.append(at[p])
            woffs += [int(v) + at[0] for v in o[1:]]
    np.testing.assert_array_equal(perm.cpu().numpy(), np.concatenate(wperm))
    np.testing.assert_array_equal(offs[: ng.value + 1].cpu().numpy(), woffs)
