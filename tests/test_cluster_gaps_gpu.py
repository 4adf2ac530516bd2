"""Grouping by gaps (cluster_by_gaps) against the oracle's sorting passes: every
split rule, field ranges whose bitmaps are refused, initial groups."""
import ctypes

import numpy as np
import pytest
import torch

from cpp_projects_b200 import _capi, cluster, search
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _cands(n, tmax, dmax, wmax, seed, base=0):
    rng = np.random.default_rng(seed)
    c = np.zeros(n, pyoracle.CAND_DTYPE)
    c["mt"] = rng.integers(0, tmax, n) + base
    c["mdt"] = rng.integers(0, dmax, n)
    c["mwidth"] = rng.integers(0, wmax, n)
    c["msnr"] = rng.integers(0, 8, n).astype(np.float32) * 0.5 + 7.0
    return c[np.lexsort((c["mwidth"], c["mt"], c["mdt"]))]


@pytest.mark.parametrize("n,tmax,dmax,wmax,metrics", [
    (1, 5, 5, 5, (2, 1, 2)), (2, 1, 1, 1, (0, 0, 0)), (3000, 4000, 70, 6, (0, 0, 0)), (3000, 4000, 70, 6, (31, 0, 1)),
    (3000, 40000, 700, 6, (32, 33, 2)), (20000, 131072, 4096, 8, (16, 8, 1 << 30)), (4000, 65, 33, 40, (1, 31, 32)),
    (5000, 5_000_000, 40, 6, (100, 1, 1)),       # more words than candidates: the sorting passes
    (2000, 300, 40, 6, (-1, 2, 1)), (2000, 300, 40, 6, (3, -1, -5)),   # negative metrics split equal values
    (100000, 3000, 900, 6, (2, 1, 2)),
])
@pytest.mark.parametrize("base", [0, -(1 << 20)])
def test_groups_members_and_delegates_match_the_oracle(cuda, n, tmax, dmax, wmax, metrics, base):
    c = _cands(n, tmax, dmax, wmax, n + tmax, base)
    perm, offs, dl = pyoracle.cluster(c, metrics)
    cl = cluster.complete_clusterization(search.cands_from_numpy(c, cuda), metrics)
    np.testing.assert_array_equal(cl.offsets.cpu().numpy(), offs)
    np.testing.assert_array_equal(cl.perm.cpu().numpy(), perm)
    np.testing.assert_array_equal(cl.delegates.cpu().numpy(), dl)


@pytest.mark.parametrize("metrics", [(16, 8, 1 << 30), (2, 1, 2), (0, 1 << 30, 0)])
def test_initial_groups_equal_clustering_each_alone(cuda, metrics):
    parts = [_cands(n, 2000, 300, 6, n) for n in (700, 0, 1, 4000, 33)]
    c = np.concatenate(parts)
    g0 = torch.from_numpy(np.repeat(np.arange(len(parts), dtype=np.int32), [len(p) for p in parts])).to(cuda)
    d = search.cands_from_numpy(c, cuda)
    n = len(c)
    perm, dl = (torch.empty(n, dtype=torch.int32, device=cuda) for _ in range(2))
    offs = torch.empty(n + 1, dtype=torch.int32, device=cuda)
    ng = ctypes.c_uint32(0)
    m = (ctypes.c_int * 3)(*metrics)
    _capi.call("bfs_cluster_grouped", d.data_ptr(), ctypes.c_uint32(n), g0.data_ptr(), ctypes.c_uint32(len(parts)), m,
               perm.data_ptr(), offs.data_ptr(), dl.data_ptr(), ctypes.byref(ng),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    wperm, woffs, at, wdl = [], [0], 0, []
    for p in parts:
        if len(p):
            a, o, k = pyoracle.cluster(p, metrics)
            wperm.append(a + at)
            woffs += [int(v) + at for v in o[1:]]
            wdl.append(k + at)
        at += len(p)
    np.testing.assert_array_equal(perm.cpu().numpy(), np.concatenate(wperm))
    np.testing.assert_array_equal(offs[: ng.value + 1].cpu().numpy(), woffs)
    # (delegates of all initial groups together are ordered by (mt, group))
    assert sorted(dl[: ng.value].cpu().numpy().tolist()) == sorted(np.concatenate(wdl).tolist())
    mt = c["mt"][dl[: ng.value].cpu().numpy()]
    assert np.all(np.diff(mt) >= 0)
