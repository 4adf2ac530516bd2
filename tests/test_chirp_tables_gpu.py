"""A chirp table counts as filled only when its kernel ran: a call that fails, or
that a stream capture merely records, leaves nothing behind that a later call reads."""
import ctypes

import pytest
import torch

from cpp_projects_b200 import _capi
from cpp_projects_b200._tensors import dev_ptr
from cpp_projects_b200.chunk import CChunk_gpu

pytestmark = pytest.mark.gpu
P = ctypes.c_void_p


@pytest.mark.parametrize("nchan,len_sft,nbin,noverlap", [(4, 8, 4096, 64),         # library transforms
                                                         (1, 2, 65536, 1024)])      # own sub-band transforms
def test_recorded_tables_are_not_filled(cuda, nchan, len_sft, nbin, noverlap):
    def chunk():
        return CChunk_gpu(1200.0, 1200.0 + 4.0 * nchan, 4, nchan, len_sft, 0, 0, 0.0, 0.0, 1, 6.0, 1, nbin, 1, noverlap,
                          0.25e-6, max_dt=8, dms=[3.0])
    ch, fresh = chunk(), chunk()
    spec = torch.randn((ch.cplx_len, 2), generator=torch.Generator(device=cuda).manual_seed(1), device=cuda)
    rows = nchan * len_sft
    want, got = torch.empty((2, rows, ch.msamp), device=cuda)
    fresh.detect_spectrum(spec, 3.0, want)
    torch.cuda.synchronize()
    rt = ctypes.CDLL("libcudart.so.12")   # (the process's own)
    s, graph = torch.cuda.Stream(), P()
    assert rt.cudaStreamBeginCapture(P(s.cuda_stream), 2) == 0
    with pytest.raises(_capi.BfsError):   # it waits for the stream, which a capture refuses
        ch.detect_spectrum(spec, 3.0, got, s)
    rt.cudaStreamEndCapture(P(s.cuda_stream), ctypes.byref(graph))
    rt.cudaGetLastError()
    torch.cuda.synchronize()
    for _ in range(3):   # (the error of the call before may be reported once more)
        try:
            ch.detect_spectrum(spec, 3.0, got)
        except _capi.BfsError:
            continue
        break
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    ch.detect_spectrum(spec, 3.0, got)    # from the table
    assert torch.equal(got, want)
