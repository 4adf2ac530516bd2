"""The coherent DM loop's preprocessing and normalisation (one mask value per
row; the mask's transform formed where it divides) against the public passes
over planes, bit for bit: the same statistics, masks, transforms and divisions."""
import ctypes

import numpy as np
import pytest
import torch

from cpp_projects_b200 import CFdmtGpu, _capi
from cpp_projects_b200.chunk import CChunk_gpu

P = ctypes.c_void_p


def _ptr(t):
    return P(t.data_ptr())


@pytest.mark.gpu
@pytest.mark.parametrize("nchan,len_sft,nbin,nfft,noverlap,max_dt,zap", [
    (4, 8, 4096, 3, 64, 16, True),       # few output rows: their columns over several CTAs
    (16, 16, 65536, 2, 1024, 256, True),
    (2, 4, 4092, 1, 36, 8, False),       # 1005 samples a row: not a multiple of four
    (8, 1, 1024, 1, 0, 1, True),
    (2, 2, 65536, 2, 512, 4, True),      # 32768-bin sub-bands: the library's own transforms
])
@pytest.mark.parametrize("npol", [2, 4])
def test_dm_loop_equals_the_separate_passes(cuda, nchan, len_sft, nbin, nfft, noverlap, max_dt, zap, npol):
    fmin, fmax, tsamp = 1200.0, 1200.0 + 4.0 * nchan, 0.25e-6
    dms = [0.0, 3.0, 7.0, 11.0, 19.0, 3.0]   # more than the kept factor tables, one of them twice
    ch = CChunk_gpu(fmin, fmax, npol, nchan, len_sft, 0, 0, 0.0, 0.0, 1, 6.0, 1, nbin, nfft, noverlap, tsamp,
                    max_dt=max_dt, dms=dms)
    g = torch.Generator(device=cuda).manual_seed(5)
    n = (nbin - 2 * noverlap) * nfft
    raw = torch.randint(-8, 8, (nchan, n, npol), generator=g, device=cuda, dtype=torch.int8)
    if zap:
        raw[0] *= 12    # its variance is far from the others': zapped (of enough rows)
    spec = ch.complex_buffer(cuda)
    for again in range(2):
        got = ch.process_raw(raw, spec)
        rows, cols = nchan * len_sft, nfft * (nbin // len_sft - 2 * (noverlap // len_sft))
        f = CFdmtGpu(fmin, fmax, rows, cols, max_dt)
        volt = ch.complex_buffer(cuda)
        for i, dm in enumerate(dms):
            plane = torch.empty((rows, cols), device=cuda)
            ch.voltages(spec, dm, volt)
            ch.detect(volt, dm, plane)
            mask, buff = torch.empty_like(plane), torch.empty(2 * rows + 4, device=cuda)
            y, norm = torch.empty((max_dt, cols), device=cuda), torch.empty((max_dt, cols), device=cuda)
            s = P(torch.cuda.current_stream().cuda_stream)
            _capi.call("bfs_preproc_calc_fdmt_inputs", _ptr(plane), rows, cols, _ptr(buff), _ptr(mask), s)
            f.process_image(mask, norm, False)
            f.process_image(plane, y, False)
            _capi.call("bfs_fdmt_normalize", _ptr(y), _ptr(norm), ctypes.c_int64(y.numel()), _ptr(y), s)
            torch.cuda.synchronize()
            assert np.array_equal(got[i].cpu().numpy().view(np.uint32), y.cpu().numpy().view(np.uint32)), (again, dm)
