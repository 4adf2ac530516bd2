"""Clustering at the edges of its sizes, against the oracle."""
import numpy as np
import pytest

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
