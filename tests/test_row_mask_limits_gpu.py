"""The channel-count form of the FDMT up to the longest delays it takes (a
histogram of the 48 KB of shared memory a kernel has), against the transform."""
import ctypes

import numpy as np
import pytest
import torch

from cpp_projects_b200 import CFdmtGpu, _capi
from cpp_projects_b200._tensors import dev_ptr
from cpp_projects_b200.chunk import CChunk_gpu

pytestmark = pytest.mark.gpu

LIMIT = 12 * 1024   # histogram entries


def _row_mask(f, mask, ncols, out):
    _capi.call("bfs_fdmt_execute_row_mask", f._plan, dev_ptr(mask), ncols, dev_ptr(out), None)


def test_row_mask_and_ones_at_the_longest_delays(cuda):
    nchan, ncols = 16, 40
    m = (np.arange(nchan) % 3 != 1).astype(np.float32)
    mask = torch.from_numpy(np.repeat(m[:, None], ncols, 1)).to(cuda)
    taken = []
    for max_dt in range(LIMIT - 6, LIMIT + 20):
        f = CFdmtGpu(1200.0, 1600.0, nchan, ncols, max_dt, fuse_depth=0, seg_levels=1)
        got, want = torch.full((2, max_dt, ncols), float("nan"), device=cuda)
        for plane, ones in ((torch.ones_like(mask), True), (mask, False)):
            f.process_image(plane, want, False)
            if ones:
                f.process_image(None, got, True)   # (beyond the limit: the transform)
            else:
                try:
                    _row_mask(f, mask, ncols, got)
                except _capi.BfsError as e:
                    assert "histogram" in str(e)
                    taken.append(False)
                    continue
                taken.append(True)
            assert torch.equal(got, want), max_dt
    # the delays pass the limit inside the range, and are taken up to there
    assert taken[0] and not taken[-1] and taken == sorted(taken, reverse=True)


def test_dm_loop_at_the_longest_delays(cuda):
    nchan, len_sft, nbin, noverlap, tsamp = 4, 4, 4096, 64, 0.25e-6
    fmin, fmax, rows, cols = 1200.0, 1216.0, 16, 1024 - 2 * 16
    plane = torch.ones((rows, cols), device=cuda)
    for max_dt in range(LIMIT + 20, LIMIT - 6, -1):   # the largest that is taken
        f = CFdmtGpu(fmin, fmax, rows, cols, max_dt, fuse_depth=0, seg_levels=1)
        y, norm = torch.empty((2, max_dt, cols), device=cuda)
        try:
            _row_mask(f, plane, cols, norm)
            break
        except _capi.BfsError as e:
            assert "histogram" in str(e)
    ch = CChunk_gpu(fmin, fmax, 2, nchan, len_sft, 0, 0, 0.0, 0.0, 1, 6.0, 1, nbin, 1, noverlap, tsamp, max_dt=max_dt, dms=[3.0])
    g = torch.Generator(device=cuda).manual_seed(5)
    raw = torch.randint(-8, 8, (nchan, nbin - 2 * noverlap, 2), generator=g, device=cuda, dtype=torch.int8)
    spec, volt = ch.complex_buffer(cuda), ch.complex_buffer(cuda)
    got = ch.process_raw(raw, spec)[0]
    ch.voltages(spec, 3.0, volt)
    ch.detect(volt, 3.0, plane)
    mask, buff = torch.empty_like(plane), torch.empty(2 * rows + 4, device=cuda)
    _capi.call("bfs_preproc_calc_fdmt_inputs", dev_ptr(plane), rows, cols, dev_ptr(buff), dev_ptr(mask), None)
    f.process_image(mask, norm, False)
    f.process_image(plane, y, False)
    _capi.call("bfs_fdmt_normalize", dev_ptr(y), dev_ptr(norm), ctypes.c_int64(y.numel()), dev_ptr(y), None)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), y.cpu().numpy().view(np.uint32))
