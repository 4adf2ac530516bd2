"""The passes of the 2^20-point forward FFT and of the 32768-point sub-band
transforms, at the edges of their dispatch.

CPU: the kernels' splits of the indices and of the twiddles, in FP64 against
numpy's FFT.  GPU: the forward FFT where the samples cannot be copied in
16-byte words (overlap or raw chunk off the word boundary), held to the 2e-6 of
the largest magnitude that the aligned form is held to; the detection of a
plane shorter than the 1024 samples between a thread's outputs, and of every
number of segments, equal to detecting the voltages (same arithmetic)."""
import numpy as np
import pytest
import torch

from cpp_projects_b200.chunk import CChunk_gpu
from oracle import chunk_oracle as co

POWERS = [1, 2, 3, 4, 8, 12, 16, 20, 24, 28]


def _w(num, den):
    return np.exp(-2j * np.pi * (np.asarray(num) % den) / den)


def _powers32(j, den):
    """w^k, k = 0..31, of w = W_den^j as the kernels form them from ten values."""
    t = dict(zip(POWERS, (_w(np.asarray(j) * k, den) for k in POWERS)))
    one = np.ones_like(t[1])
    return np.stack([(t[4 * (k // 4)] if k >= 4 else one) * (t[k % 4] if k % 4 else one) for k in range(32)])


def _fft1024(v, first):
    """(1024, m): two 32-point steps, first = factors (32 m1, 32 b, m or 1) between them."""
    m = v.shape[1]
    u = np.fft.fft(v.reshape(32, 32, m), axis=0) * first       # over a: [m1][b]
    return np.transpose(np.fft.fft(u, axis=1), (1, 0, 2)).reshape(1024, m)   # over b: [m2][m1]


def test_forward_passes_index_math():
    n = 1 << 20
    rng = np.random.default_rng(0)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a = x.reshape(1024, 1024)                                   # [n1][n2]
    b, n2 = np.arange(32)[:, None], np.arange(1024)[None, :]
    cols = _fft1024(a, _powers32(1024 * b + n2, n))             # [k1][n2], the m1 part of the twiddles included
    k1 = np.arange(1024)[:, None]
    cols = cols * _w(n2 * (k1 // 32), 32768)                    # the row pass's factor
    rows = _fft1024(cols.T, _powers32(np.arange(32)[:, None], 1024))
    want = np.fft.fft(x)
    assert np.abs(rows.reshape(-1) - want).max() < 1e-11 * np.abs(want).max()


def test_subband_passes_index_math():
    rng = np.random.default_rng(1)
    y = rng.standard_normal(32768) + 1j * rng.standard_normal(32768)
    z = np.fft.fft(y.reshape(32, 1024), axis=0) * _powers32(np.arange(1024), 32768)   # [q][b]
    out = _fft1024(z.T, _powers32(np.arange(32)[:, None], 1024))                      # [p][q]
    want = np.fft.fft(y)
    assert np.abs(out.reshape(-1) - want).max() < 1e-12 * np.abs(want).max()


def _make(cuda, npol=4, nchan=2, len_sft=32, nbin=1 << 20, nfft=2, noverlap=8192, seed=1):
    fmax = 1200.0 + 16.0 * nchan
    ch = CChunk_gpu(1200.0, fmax, npol, nchan, len_sft, 0, 0, 0.0, 0.0, 1, 6.0, 1, nbin, nfft, noverlap,
                    1.0 / 16.0 * 1e-6, max_dt=4, dms=[0.0])
    g = co.Geometry(fmin=1200.0, fmax=fmax, npol=npol, nchan=nchan, len_sft=len_sft, nbin=nbin, nfft=nfft,
                    noverlap=noverlap, tsamp=1.0 / 16.0 * 1e-6, max_dt=4)
    raw = np.random.default_rng(seed).integers(-128, 128, size=(g.nchan, g.len_chunk, g.npol), dtype=np.int8)
    return ch, g, raw


@pytest.mark.gpu
@pytest.mark.parametrize("npol,noverlap,offset", [(4, 8192, 0), (4, 8194, 0), (4, 8191, 0), (4, 8192, 4), (4, 0, 8),
                                                  (2, 8200, 0), (2, 8196, 0), (2, 8193, 0), (2, 8192, 2)])
def test_forward_fft_of_samples_on_and_off_the_word_boundary(cuda, npol, noverlap, offset):
    ch, g, raw = _make(cuda, npol=npol, noverlap=noverlap, nchan=1)
    buf = torch.zeros(raw.size + 16, dtype=torch.int8, device=cuda)
    d_raw = buf[offset:offset + raw.size].view(raw.shape)
    d_raw.copy_(torch.from_numpy(raw))
    spec = ch.complex_buffer(cuda)
    ch.unpack_fft(d_raw, spec)
    got = spec.cpu().numpy().view(np.complex64).reshape(g.npol // 2, g.nfft, g.nchan, g.nbin)
    want = np.fft.fft(co.unpack(g, raw).astype(np.complex128), axis=-1)
    assert np.abs(got - want).max() < 2e-6 * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("npol,nfft,noverlap", [(4, 1, 32000), (2, 1, 32640), (4, 3, 512), (2, 2, 0), (4, 2, 32766)])
def test_detection_equals_detect_of_voltages(cuda, npol, nfft, noverlap):
    ch, g, raw = _make(cuda, npol=npol, nchan=3, len_sft=2, nbin=65536, nfft=nfft, noverlap=noverlap)
    d = ch.complex_buffer(cuda)
    ch.unpack(torch.from_numpy(raw).to(cuda), d)
    ch.forward_fft(d)
    for dm in (0.0, 40.0):
        v = ch.complex_buffer(cuda)
        ch.voltages(d, dm, v)
        got = v.cpu().numpy().view(np.complex64).reshape(g.npol // 2, g.nfft, g.nchan, g.nbin)
        want = co.voltages(g, d.cpu().numpy().view(np.complex64).reshape(got.shape).astype(np.complex128), dm)
        assert np.abs(got - want).max() < 1e-5 * np.abs(want).max()
        plane = torch.full((2, g.rows, g.msamp), float("nan"), device=cuda)
        ch.detect(v, dm, plane[0])
        ch.detect_spectrum(d, dm, plane[1])
        assert torch.equal(plane[0].view(torch.int32), plane[1].view(torch.int32))
