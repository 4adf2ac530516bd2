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
@pytest.mark.parametrize("nchan", [64, 100, 256, 512, 1024])
def test_tuned_16bit_plans_are_measured(cuda, prec, nchan):
    depths = []
    for ncols in (1500, 700, 300, 40000):   # (measured once each: the lengths' cache entries differ)
        d = _capi.FdmtDesc(**BAND, nchan=nchan, ncols=ncols, max_dt=nchan, precision=prec)
        t, ms = autotune_desc(d)
        assert 0.0 < ms < 1e3
        f = CFdmtGpu(1200.0, 1600.0, nchan, ncols, nchan, fuse_depth=-2, precision=prec)
        own = (f.info.fuse_depth, f.info.hbm_passes, f.info.seg_levels)
        assert own == info_of(t) == info_of(t, host=True) and own[0] == t.fuse_depth
        depths.append(own[0])
    # a level of a short plane costs a launch and the head forms several in one: depth 2 to 5
    # wherever it was measured
    assert max(depths[:3]) >= 2


LOW = ((400.0, 800.0), (110.0, 190.0))
SHAPES = [(1200.0, 1600.0, n, m) for n, m in ((4096, 2048), (4096, 1024), (2048, 1024), (1024, 512), (1024, 256),
                                              (256, 64), (128, 32), (1024, 1024))] + \
         [(*b, 1024, 256) for b in LOW]


@pytest.mark.parametrize("fmin,fmax,nchan,max_dt", SHAPES)
@pytest.mark.parametrize("levels", [0, 4, 3, 2])
def test_run_segment_schedules_can_be_created(fmin, fmax, nchan, max_dt, levels):
    """Every schedule of run segments the autotuner may choose, and the default's, as the same passes."""
    d = _capi.FdmtDesc(fmin=fmin, fmax=fmax, nchan=nchan, ncols=4000, max_dt=max_dt, seg_levels=levels,
                       fuse_depth=0 if levels else -1)
    most, niter = levels or 4, nchan.bit_length() - 1
    depth, passes, got = info_of(d, host=True)
    assert (depth, passes) == (0, -(-niter // most)) and got <= most
    plan, n, pp = ctypes.c_void_p(), ctypes.c_int(0), (ctypes.c_int * (13 * passes))()
    _capi.call("bfs_fdmt_plan_create_host", ctypes.byref(d), ctypes.byref(plan))
    _capi.call("bfs_fdmt_plan_passes", plan, ctypes.byref(n), pp, len(pp))
    _capi.lib().bfs_fdmt_plan_destroy(plan)
    assert pp[12] > 0   # the first pass reads the channels


@pytest.mark.gpu
@pytest.mark.parametrize("fmin,fmax,nchan,max_dt", SHAPES + [(1200.0, 1600.0, n, n) for n in (4, 8, 16)])
def test_tuned_plans_time_the_default_schedule(cuda, fmin, fmax, nchan, max_dt):
    passes = []
    for ncols in (1000, 500, 250):   # (measured once each: the lengths' cache entries differ)
        d = _capi.FdmtDesc(fmin=fmin, fmax=fmax, nchan=nchan, ncols=ncols, max_dt=max_dt)
        t, ms = autotune_desc(d)
        assert 0.0 < ms < 1e3
        f = CFdmtGpu(fmin, fmax, nchan, ncols, max_dt, fuse_depth=-2)
        own = (f.info.fuse_depth, f.info.hbm_passes, f.info.seg_levels)
        assert own == info_of(t) == info_of(t, host=True)
        passes.append(own[1])
    # a short plane's passes cost a launch each: no more of them than the default's
    assert min(passes) <= -(-(nchan.bit_length() - 1) // 4)


@pytest.mark.gpu
@pytest.mark.parametrize("nchan", [2, 4, 8, 16, 64])
def test_tuned_pravir_plans_are_measured(cuda, nchan):
    d = _capi.FdmtDesc(**BAND, nchan=nchan, ncols=1000, max_dt=nchan, plan_kind=1, tsamp=1e-3)
    t, ms = autotune_desc(d)
    assert 0.0 < ms < 1e3
    assert info_of(t)[:2] == info_of(t, host=True)[:2]
