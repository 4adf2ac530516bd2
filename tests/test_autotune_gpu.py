"""The autotuner measures every kind of plan, and the description it returns is the schedule it runs."""
import ctypes

import pytest

from cpp_projects_b200 import CFdmtGpu, _capi
from cpp_projects_b200.fdmt import autotune_desc

BAND = dict(fmin=1200.0, fmax=1600.0)


def info_of(desc, host=False):
    plan, info = ctypes.c_void_p(), _capi.FdmtInfo()
    _capi.call("bfs_fdmt_plan_create_host" if host else "bfs_fdmt_plan_create", ctypes.byref(desc), ctypes.byref(plan))
    try:
        _capi.call("bfs_fdmt_plan_info", plan, ctypes.byref(info))
        return info.fuse_depth, info.hbm_passes, info.seg_levels
    finally:
        _capi.lib().bfs_fdmt_plan_destroy(plan)


@pytest.mark.parametrize("levels", [0, 1])
def test_run16_flag(levels):
    """An explicit depth 0 of a 16-bit plan: plain passes, run segments with the flag."""
    d = _capi.FdmtDesc(**BAND, nchan=256, ncols=3000, max_dt=256, precision=1, seg_levels=levels)
    assert info_of(d, host=True) == (0, 8, 1)
    d.seg_flags = _capi.BFS_SEG_RUN16
    if levels == 0:
        assert info_of(d, host=True) == (0, 2, 4)
        d.precision = 0
    with pytest.raises(_capi.BfsError):
        info_of(d, host=True)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("nchan,ncols", [(64, 1500), (256, 1500), (512, 4000), (100, 3000), (1024, 40000)])
def test_tuned_16bit_plans_are_measured(cuda, prec, nchan, ncols):
    d = _capi.FdmtDesc(**BAND, nchan=nchan, ncols=ncols, max_dt=nchan, precision=prec)
    t, ms = autotune_desc(d)
    assert 0.0 < ms < 1e3
    # a level of a short plane costs a launch, the head forms several in one: depth 2 to 5
    # wherever it was measured up to 512 channels and 4000 samples
    assert t.fuse_depth >= 2 or ncols > 4000
    f = CFdmtGpu(1200.0, 1600.0, nchan, ncols, nchan, fuse_depth=-2, precision=prec)
    own = (f.info.fuse_depth, f.info.hbm_passes, f.info.seg_levels)
    assert own == info_of(t) == info_of(t, host=True) and own[0] == t.fuse_depth
