// Forward FFT of the 2^20-sample coherent-dedispersion segments, fused with
// the GUPPI unpack (sm_100a).
//
// The reference unpacks the int8 chunk into a complex buffer
// (unpack_chunk_guppi_gpu, L/CDMT/Session_guppi_gpu.cu:117-141) and then runs
// cuFFT's C2C forward transform of length nbin on every (pol, fft, channel)
// segment (CChunk_gpu::process, L/CDMT/Chunk_gpu.cu:267).  Here, for
// nbin = 2^20, the two steps are two kernels of a four-step transform
// (N = N1 N2, N1 = N2 = 1024; n = n1 N2 + n2, k = k2 N1 + k1):
//   column pass  B[k1][n2] = W_N^(n2 (k1 mod 32)) sum_n1 x[n1 N2 + n2] W_N1^(n1 k1),
//                with x read straight from the int8 samples (overlap-save
//                zeros included), both polarisations of a sample at once;
//   row pass     X[k2 N1 + k1] = sum_n2 B[k1][n2] W_N^(n2 (k1 - k1 mod 32)) W_N2^(n2 k2),
//                written in natural order.
// A 1024-point transform is two 32-point radix-2 transforms in registers with
// a twiddle W_1024^(b m1) and an exchange through shared memory between them;
// a CTA runs eight.  Twiddles come from small tables rounded once from FP64
// (products of two table values where a full table would not fit on chip).
// The result agrees with the unpack + cuFFT form to FP32 rounding (it is not
// bit-identical: a different FFT).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "internal.h"
#include "row_ops.cuh"

namespace bfs {
namespace {

constexpr int kF = 1024;          // both factors of the four-step transform
constexpr long long kFftN = static_cast<long long>(kF) * kF;
constexpr int kTile = 33;         // padded row of a 32 x 32 exchange tile
constexpr int kRegion = 32 * kTile + 2;  // float2 per tile (the +2 staggers the tiles' banks)
constexpr int kCols = 8;          // columns per CTA in the column pass
constexpr int kColPitch = 32 * kCols + 8;  // float2 per exchanged row of the column pass (the +8 staggers the rows' banks)
constexpr int kRows = 8;          // rows per CTA in the row pass (64-byte output runs)
constexpr int kSubN = 32 * kF;    // sub-band transforms of the coherent stage (mbin = 32768)

// cos(pi k / 16), k = 0..8, each rounded once to float (sin(pi k/16) = cos16(8-k)).
__host__ __device__ constexpr float cos16(int k) {
    return k == 0 ? 1.0f : k == 1 ? 0x1.f6297cp-1f : k == 2 ? 0x1.d906bcp-1f : k == 3 ? 0x1.a9b662p-1f
         : k == 4 ? 0x1.6a09e6p-1f : k == 5 ? 0x1.1c73b4p-1f : k == 6 ? 0x1.87de2ap-2f
         : k == 7 ? 0x1.8f8b84p-3f : 0.0f;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// d * W_32^k, W_32 = exp(-2 pi i / 32), k = 0..15 a compile-time constant
// after unrolling (k = 0 and 8 exact).
__device__ __forceinline__ float2 tw32(float2 d, int k) {
    if (k == 0) return d;
    if (k == 8) return make_float2(d.y, -d.x);
    const float2 w = k < 8 ? make_float2(cos16(k), -cos16(8 - k)) : make_float2(-cos16(16 - k), -cos16(k - 8));
    return cmul(d, w);
}

__host__ __device__ constexpr int bitrev5(int k) {
    return ((k & 1) << 4) | ((k & 2) << 2) | (k & 4) | ((k & 8) >> 2) | ((k & 16) >> 4);
}

// a + b and a - b, both halves in one instruction, each rounded to nearest.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
    float2 o;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(o.x), "=f"(o.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return o;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
    float2 o;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(o.x), "=f"(o.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return o;
}

// In-place 32-point forward DFT of r (decimation in frequency): afterwards
// X[k] = r[bitrev5(k)].
__device__ __forceinline__ void dft32(float2 (&r)[32]) {
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
#pragma unroll
        for (int g = 0; g < 32; g += 2 * h) {
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const float2 a = r[g + j], b = r[g + j + h];
                r[g + j] = cadd(a, b);
                r[g + j + h] = tw32(csub(a, b), j * (16 / h));
            }
        }
    }
}

// r[bitrev5(k)] *= w^k for k = 0..31, where the ten values w^1, w^2, w^3, w^4,
// w^8, ... w^28 stand at t[0], t[stride], ...: w^(4 a + c) is one product of
// two values, each rounded once.
__device__ __forceinline__ void twiddle32(float2 (&r)[32], const float2* __restrict__ t, int stride) {
    float2 wc[4];
#pragma unroll
    for (int c = 1; c < 4; ++c) wc[c] = __ldg(t + (c - 1) * stride);
#pragma unroll
    for (int c = 1; c < 4; ++c) r[bitrev5(c)] = cmul(r[bitrev5(c)], wc[c]);
#pragma unroll
    for (int a = 1; a < 8; ++a) {
        const float2 wa = __ldg(t + (2 + a) * stride);
        r[bitrev5(4 * a)] = cmul(r[bitrev5(4 * a)], wa);
#pragma unroll
        for (int c = 1; c < 4; ++c) r[bitrev5(4 * a + c)] = cmul(r[bitrev5(4 * a + c)], cmul(wa, wc[c]));
    }
}

// The int8 pair of polarisation pol of a sample as floats: the bytes, offset
// by 128, become the low mantissa bits of 2^23, so that one exact subtraction
// of 2^23 + 128 leaves their values.
__device__ __forceinline__ float2 int8_pair(int v, int pol) {
    const unsigned u = static_cast<unsigned>(v) ^ 0x80808080u;
    const unsigned sel = pol ? 0x7652u : 0x7650u;   // byte 2 pol under the upper bytes of 2^23
    const float re = __uint_as_float(__byte_perm(u, 0x4b000000u, sel));
    const float im = __uint_as_float(__byte_perm(u, 0x4b000000u, sel + 1));
    return csub(make_float2(re, im), make_float2(8388736.0f, 8388736.0f));
}

// 1024-point transforms are two 32-point steps, u = 32 a + b and
// v = m1 + 32 m2 (a, b, m1, m2 < 32): over a, times W_1024^(b m1), an exchange
// through shared memory, over b.  A CTA of 256 threads runs eight of them, and
// the two steps use different threads' shapes: where a side has the transform's
// values contiguous in memory, a warp is one transform's 32 values of b (m1);
// where it has the eight transforms side by side, a warp is four values of
// b (m1) of all eight, so that loads and stores go straight between registers
// and memory in runs of eight values and nothing is staged for their sake.

// Rows in, runs of eight out: r[a] = v[32 a + lane] of transform t = warp on
// entry; on exit V[m1 + 32 m2] of transform t = threadIdx.x % 8 in
// r[bitrev5(m2)], m1 = threadIdx.x / 8.  sm: 8 kRegion.
__device__ __forceinline__ void fft1024_rows(float2 (&r)[32], float2* __restrict__ sm,
                                             const float2* __restrict__ tw) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    dft32(r);
    twiddle32(r, tw + lane, 32);
    float2* out = sm + w * kRegion + lane * kTile;
#pragma unroll
    for (int m1 = 0; m1 < 32; ++m1) out[m1] = r[bitrev5(m1)];
    __syncthreads();
    const float2* in = sm + (threadIdx.x & 7) * kRegion + (threadIdx.x >> 3);
#pragma unroll
    for (int b = 0; b < 32; ++b) r[b] = in[b * kTile];
    dft32(r);
}

// Column pass.  grid (kF / kCols, nfft, nchan); NP2 polarisations, one after
// the other.  The result lacks the factor W_32768^(n2 (k1 / 32)) of its
// twiddles, which the row pass has time for.  The samples are staged in shared memory
// ([n1][c]); thread (b, c), c fastest, of the first step has the samples
// n1 = 32 a + b of column c0 + c, thread (m1, c) of the second the results
// k1 = m1 + 32 m2.  VEC: the kCols samples of every n1 are whole 16-byte words
// of the chunk, each inside it or outside it; else samples one by one.
//
// Bound by instruction issue and the latency of its phases at 16 warps per SM
// (46 % of the issue slots; 24 warps do not fit in the registers without
// spilling and are slower).  4 x 32 segments of 2^20, two polarisations: 643 us;
// 1208 us with samples and results staged per warp for runs of four columns
// (LSU pipe 78 % busy), 746 us with the row pass's factor applied here, 812 us
// with 4-byte sample loads straight to registers, 754 us with the next group's
// samples copied during this one's second step.
template <int NP2, bool VEC>
__global__ void __launch_bounds__(32 * kCols, 2)
k_fft_cols_guppi(const signed char* __restrict__ raw, float2* __restrict__ y, const float2* __restrict__ twa,
                 long long nsamp, int noverlap, int nfft, int nchan) {
    using Sample = std::conditional_t<NP2 == 2, int, short>;   // bytes re0, im0, re1, im1
    constexpr int kPerWord = 16 / static_cast<int>(sizeof(Sample));
    constexpr int kWords = kCols / kPerWord;                   // words of one n1
    constexpr int kThreads = 32 * kCols;
    extern __shared__ __align__(16) float2 sm_cols[];
    Sample* stage = reinterpret_cast<Sample*>(sm_cols + 32 * kColPitch);
    const int c0 = blockIdx.x * kCols, ifft = blockIdx.y, ichan = blockIdx.z;
    const int c = threadIdx.x % kCols, h = threadIdx.x / kCols;   // h: b, then m1
    const long long first = static_cast<long long>(kFftN - 2 * noverlap) * ifft - noverlap;   // sample of n = 0
    const Sample* chan = reinterpret_cast<const Sample*>(raw) + static_cast<long long>(ichan) * nsamp;
    if constexpr (VEC) {
        const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(stage));
#pragma unroll
        for (int k = 0; k < kF * kWords / kThreads; ++k) {
            const int e = threadIdx.x + k * kThreads;
            const long long isamp = first + (e / kWords) * kF + c0 + (e % kWords) * kPerWord;
            if (isamp >= 0 && isamp < nsamp) copy16(dst + 16 * e, chan + isamp);
            else *reinterpret_cast<int4*>(stage + kPerWord * e) = make_int4(0, 0, 0, 0);
        }
        copy_wait();
    } else {
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
            const long long isamp = first + (h + 32 * k) * kF + c0 + c;
            stage[threadIdx.x + k * kThreads] = isamp >= 0 && isamp < nsamp ? __ldg(chan + isamp) : 0;
        }
    }
#pragma unroll 1
    for (int p = 0; p < NP2; ++p) {
        __syncthreads();   // the samples have arrived; the last polarisation's exchange is read
        float2 r[32];
#pragma unroll
        for (int a = 0; a < 32; ++a) r[a] = int8_pair(stage[threadIdx.x + a * kThreads], p);
        dft32(r);
        twiddle32(r, twa + h * kF + c0 + c, kSubN);   // W_1024^(b m1) W_N^(n2 m1) = W_N^((1024 b + n2) m1)
#pragma unroll
        for (int m1 = 0; m1 < 32; ++m1) sm_cols[h * kColPitch + m1 * kCols + c] = r[bitrev5(m1)];
        __syncthreads();
#pragma unroll
        for (int b = 0; b < 32; ++b) r[b] = sm_cols[b * kColPitch + threadIdx.x];
        dft32(r);
        float2* out = y + ((static_cast<size_t>(p) * nfft + ifft) * nchan + ichan) * kFftN + h * kF + c0 + c;
#pragma unroll
        for (int m2 = 0; m2 < 32; ++m2) out[m2 * 32 * kF] = r[bitrev5(m2)];
    }
}

// Row pass.  grid (kF / kRows, segments); warp w reads row r0 + w, completes its
// twiddles (one row of twb per CTA: r0 / 32 is k1 / 32 of all its rows) and
// the CTA writes X[k2 N1 + r0 .. + kRows).
//
// Bound by HBM: 4 x 32 segments, two polarisations, 4.3 GB in 750 us (5.7
// TB/s); 822 us with four rows per CTA staged for the stores (LSU pipe 86 %
// busy).
__global__ void __launch_bounds__(32 * kRows, 2)
k_fft_rows(const float2* __restrict__ y, float2* __restrict__ x, const float2* __restrict__ tw,
           const float2* __restrict__ twb) {
    extern __shared__ float2 sm_rows[];
    const int r0 = blockIdx.x * kRows;
    const size_t seg = blockIdx.y;
    const float2* row = y + seg * kFftN + static_cast<size_t>(r0 + (threadIdx.x >> 5)) * kF + (threadIdx.x & 31);
    float2 r[32];
#pragma unroll
    for (int a = 0; a < 32; ++a) r[a] = __ldg(row + 32 * a);
    const float2* wb = twb + (r0 / 32) * kF + (threadIdx.x & 31);
#pragma unroll
    for (int a = 0; a < 32; ++a) r[a] = cmul(r[a], __ldg(wb + 32 * a));
    fft1024_rows(r, sm_rows, tw);
    float2* out = x + seg * kFftN + static_cast<size_t>(threadIdx.x / kRows) * kF + r0 + threadIdx.x % kRows;
#pragma unroll
    for (int m2 = 0; m2 < 32; ++m2) out[m2 * 32 * kF] = r[bitrev5(m2)];
}

// ---- inverse sub-band transforms of the coherent stage ------------------------
// Every mbin = 32768-sample sub-band of the chirped spectrum is transformed
// back (CChunk_fly_gpu::elementWiseMult + the inverse cufftExecC2C of
// CChunk_gpu::process, L/CDMT/Chunk_fly_gpu.cu:94-163, Chunk_gpu.cu:288-290).
// v = IDFT(x) is computed as conj(DFT(conj(x))), the forward DFT of
// y = conj(chirp x) by four steps with m = 1024 a + b (a < 32, b < 1024) and
// n = q + 32 p (q < 32, p < 1024):
//   pass A  Z[q][b] = W_N^(b q) sum_a y[1024 a + b] W_32^(a q)   (one thread per b)
//   pass B  Y[q + 32 p] = sum_b Z[q][b] W_1024^(b p)               (one warp per q)
// and v = conj(Y).  The 32-point step comes first: its threads read and write
// whole lines of the spectrum and of Z and exchange nothing, and each warp of
// the 1024-point step reads one contiguous row.  The chirp is read from a
// per-DM table of the factors k_chirp applies (the same FP32 products), so
// the FP64 phase is evaluated once per (channel, sub-band, bin), not once per
// polarisation and FFT segment.  Pass A stores Z in the sub-band's own place
// (Z[q][b] at offset 1024 q + b).  Pass B detects: |v|^2 / nbin^2 summed over
// the polarisations, rolled, unpadded, reversed and shifted as k_detect does,
// straight into the dedispersed plane; or it writes v over Z, the four CTAs
// of a sub-band as one cluster that has read all of Z before any of it
// writes.
constexpr int kSubThreads = 128;         // pass A: values of b per CTA
constexpr int kSubQ = 8;                 // pass B: values of q per CTA
constexpr size_t kSubSmem = sizeof(float2) * kSubQ * kRegion;

// Bounds: pass A is HBM-bound (4 x 32 segments of 32 sub-bands, two
// polarisations: 685 us for 4.6 GB, 6.7 TB/s; 1153 us as the 1024-point
// transforms of eight interleaved columns; 772 us at 16 warps per SM, which
// spill, instead of 12).  Pass B is bound by issue (51 %) and its phases' latency at 16
// warps: 600 us, of which 2.6 GB of memory traffic account for 400 (the
// 32-point form it replaces: 642 us); with the powers staged for the stores
// 609 us, 24 warps 939 us (spills).

// Pass A.  blockIdx.x = block of b + 8 (fft + nfft (sub-band + len_sft chan)):
// the CTAs that share a block of the chirp table are neighbours.
__global__ void __launch_bounds__(kSubThreads, 3)
k_subfft_cols(const float2* __restrict__ spec, const float2* __restrict__ chirp, float2* __restrict__ z,
              const float2* __restrict__ tws, int npol2, int nfft, int nchan, int len_sft, int nbin) {
    constexpr int kBlk = kF / kSubThreads;
    int id = blockIdx.x;
    const int b = (id % kBlk) * kSubThreads + threadIdx.x;
    id /= kBlk;
    const int f = id % nfft, sub = id / nfft;
    const int ichan = sub / len_sft, isft = sub % len_sft;
    const int chunk = (isft + len_sft / 2) % len_sft;   // fft-shifted place of the sub-band
    const float2* ch = chirp + static_cast<size_t>(sub) * kSubN + b;
    for (int p = 0; p < npol2; ++p) {
        const size_t base = ((static_cast<size_t>(p) * nfft + f) * nchan + ichan) * nbin +
                            static_cast<size_t>(chunk) * kSubN + b;
        float2 r[32];
#pragma unroll
        for (int a = 0; a < 32; ++a) r[a] = __ldg(spec + base + static_cast<size_t>(a) * kF);
#pragma unroll
        for (int a = 0; a < 32; ++a) {
            // y = conj(x * chirp), the product as k_chirp forms it
            const float2 c = __ldg(ch + a * kF);
            const float ox = __fsub_rn(__fmul_rn(r[a].x, c.x), __fmul_rn(r[a].y, c.y));
            const float oy = __fadd_rn(__fmul_rn(r[a].x, c.y), __fmul_rn(r[a].y, c.x));
            r[a] = make_float2(ox, -oy);
        }
        dft32(r);
        twiddle32(r, tws + b, kF);   // W_32768^(b q)
#pragma unroll
        for (int q = 0; q < 32; ++q) z[base + static_cast<size_t>(q) * kF] = r[bitrev5(q)];
    }
}

// Pass B.  blockIdx.x = block of q + 4 (sub-band + len_sft (chan + nchan outer)):
// outer = fft (DETECT: both polarisations) or segment.  Warp w reads the row
// q = 8 block + w; thread (m1, qq), qq fastest, has the results
// n = 8 block + qq + 32 (m1 + 32 m2).
template <bool DETECT>
__global__ void __launch_bounds__(32 * kSubQ, 2)
k_subfft_rows(float2* __restrict__ z, float* __restrict__ plane, const int* __restrict__ shift,
              const float2* __restrict__ tw, int npol2, int nfft, int nchan, int len_sft, int nbin, int nov_pc,
              int mbin_adj, int msamp, double inv_nbin2) {
    constexpr int kBlk = 32 / kSubQ;
    extern __shared__ float2 sm_sub[];
    int id = blockIdx.x;
    const int q0 = (id % kBlk) * kSubQ;
    id /= kBlk;
    const int isft = id % len_sft;
    id /= len_sft;
    const int ichan = id % nchan, outer = id / nchan;
    const size_t sub_off = static_cast<size_t>((isft + len_sft / 2) % len_sft) * kSubN;
    const int in = (q0 + (threadIdx.x >> 5)) * kF + (threadIdx.x & 31);
    const int n0 = q0 + threadIdx.x % kSubQ + 32 * (threadIdx.x / kSubQ);   // m2 = 0
    float2 r[32];
    if constexpr (!DETECT) {
        float2* zz = z + (static_cast<size_t>(outer) * nchan + ichan) * nbin + sub_off;
#pragma unroll
        for (int a = 0; a < 32; ++a) r[a] = zz[in + 32 * a];
        // every CTA of the sub-band has read its rows before any writes over them
        cooperative_groups::this_cluster().sync();
        fft1024_rows(r, sm_sub, tw);
#pragma unroll
        for (int m2 = 0; m2 < 32; ++m2) {
            const float2 y = r[bitrev5(m2)];
            zz[n0 + kF * m2] = make_float2(y.x, -y.y);
        }
    } else {
        float acc[32];
#pragma unroll
        for (int m2 = 0; m2 < 32; ++m2) acc[m2] = 0.0f;
        for (int p = 0; p < npol2; ++p) {
            const float2* zz = z + ((static_cast<size_t>(p) * nfft + outer) * nchan + ichan) * nbin + sub_off + in;
#pragma unroll
            for (int a = 0; a < 32; ++a) r[a] = __ldg(zz + 32 * a);
            if (p) __syncthreads();   // the last polarisation's exchange is read
            fft1024_rows(r, sm_sub, tw);
#pragma unroll
            for (int m2 = 0; m2 < 32; ++m2) {
                // |v|^2 / nbin / nbin in FP64 (x^2 and y^2 of floats are exact in
                // double; nbin a power of two: the scaling is exact), then FP32
                const float2 y = r[bitrev5(m2)];
                const double px = y.x, py = y.y;
                acc[m2] = __fadd_rn(acc[m2], static_cast<float>((px * px + py * py) * inv_nbin2));
            }
        }
        const int row = (nchan - 1 - ichan) * len_sft + (len_sft - 1 - isft);
        float* out = plane + static_cast<size_t>(row) * msamp;
        const long long to = (static_cast<long long>(outer) * mbin_adj + (n0 - nov_pc) + __ldg(shift + row)) % msamp;
        int col = static_cast<int>(to < 0 ? to + msamp : to);
        const int step = kF % msamp;
#pragma unroll
        for (int m2 = 0; m2 < 32; ++m2) {
            const int n = n0 + kF * m2;
            if (n >= nov_pc && n < nov_pc + mbin_adj) out[col] = acc[m2];
            col += step;
            if (col >= msamp) col -= msamp;
        }
    }
}

constexpr size_t kColSmem(int npol) { return sizeof(float2) * 32 * kColPitch + static_cast<size_t>(npol) * kF * kCols; }
constexpr size_t kRowSmem = sizeof(float2) * static_cast<size_t>(kRows) * kRegion;

// Twiddle tables of one device, each value rounded once from FP64.  tw, tws
// and twa hold the ten powers of twiddle32: of W_1024^lane, of W_32768^b
// (b < 1024) and of W_N^j (j < 32768); twb[m2][n2] = W_32768^(n2 m2).
struct FftTables {
    float2* tw = nullptr;
    float2* tws = nullptr;
    float2* twa = nullptr;
    float2* twb = nullptr;
};
std::mutex g_fft_mu;
std::vector<FftTables> g_fft_tables;

bfs_status fft_tables(FftTables* out) {
    int dev = 0;
    BFS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_fft_mu);
    if (static_cast<int>(g_fft_tables.size()) <= dev) g_fft_tables.resize(dev + 1);
    FftTables& t = g_fft_tables[dev];
    if (!t.tw) {
        const double pi = 3.14159265358979323846;
        auto w = [&](long long num, long long den) {
            const double ph = -2.0 * pi * static_cast<double>(num % den) / static_cast<double>(den);
            return make_float2(static_cast<float>(std::cos(ph)), static_cast<float>(std::sin(ph)));
        };
        std::vector<float2> all;
        auto powers = [&](int count, long long den) {
            for (int k : {1, 2, 3, 4, 8, 12, 16, 20, 24, 28})
                for (long long b = 0; b < count; ++b) all.push_back(w(b * k, den));
        };
        powers(32, kF);
        const size_t at_tws = all.size();
        powers(kF, kSubN);
        const size_t at_a = all.size();
        powers(kSubN, kFftN);
        const size_t at_b = all.size();
        for (long long m = 0; m < 32; ++m)
            for (long long n2 = 0; n2 < kF; ++n2) all.push_back(w(n2 * m, kSubN));
        float2* d = nullptr;
        BFS_CUDA(cudaMalloc(&d, all.size() * sizeof(float2)));
        const cudaError_t e = cudaMemcpy(d, all.data(), all.size() * sizeof(float2), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) { cudaFree(d); return fail(BFS_ERR_CUDA, "FFT twiddle upload: %s", cudaGetErrorString(e)); }
        t.tw = d;
        t.tws = d + at_tws;
        t.twa = d + at_a;
        t.twb = d + at_b;
    }
    *out = t;
    return BFS_OK;
}

template <typename K>
bfs_status smem_opt_in(K kern, size_t bytes) {
    static std::mutex mu;
    static std::vector<std::pair<const void*, int>> done;
    int dev = 0;
    BFS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    for (const auto& d : done)
        if (d.first == reinterpret_cast<const void*>(kern) && d.second == dev) return BFS_OK;
    BFS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
    done.emplace_back(reinterpret_cast<const void*>(kern), dev);
    return BFS_OK;
}

}  // namespace

bool fft_fused_supported(int nbin, int npol) { return nbin == kFftN && (npol == 2 || npol == 4); }

// The own sub-band transforms: mbin = nbin / len_sft = 32768, nbin a power of
// two, one or two polarisations.
bool subband_ifft_supported(int nbin, int len_sft, int npol) {
    return len_sft >= 1 && nbin % len_sft == 0 && nbin / len_sft == kSubN && (nbin & (nbin - 1)) == 0 &&
           (npol == 2 || npol == 4);
}

// Inverse transforms of every chirped sub-band of spec (complex64
// [pol][fft][chan][nbin], 16-byte aligned) with the chirp table chirp
// ([chan][sub-band][mbin], 16-byte aligned): plane == nullptr -> the voltages
// in z (same layout as spec); else z is scratch and the detected,
// dedispersed plane (rows x msamp) goes to plane, shift = the rows' shifts.
bfs_status subband_ifft(const float2* spec, const float2* chirp, float2* z, float* plane, const int* shift,
                        int npol2, int nfft, int nchan, int len_sft, int nbin, int nov_pc, int mbin_adj, int msamp,
                        cudaStream_t s) {
    FftTables t;
    bfs_status st = fft_tables(&t);
    if (st != BFS_OK) return st;
    BFS_ARG(subband_ifft_supported(nbin, len_sft, 2 * npol2), "no own sub-band transform for this geometry");
    BFS_ARG(reinterpret_cast<uintptr_t>(spec) % 16 == 0 && reinterpret_cast<uintptr_t>(chirp) % 16 == 0,
            "spectrum and chirp table must be 16-byte aligned");
    const long long nseg = static_cast<long long>(npol2) * nfft;
    const long long nsub = static_cast<long long>(nchan) * len_sft;
    constexpr int kBlkA = kF / kSubThreads, kBlkB = 32 / kSubQ;
    BFS_ARG(kBlkA * nseg * nsub < (1ll << 31), "too many sub-bands");
    k_subfft_cols<<<static_cast<unsigned>(kBlkA * nfft * nsub), kSubThreads, 0, s>>>(
        spec, chirp, z, t.tws, npol2, nfft, nchan, len_sft, nbin);
    BFS_LAUNCH_CHECK("k_subfft_cols");
    const double inv_nbin2 = 1.0 / (static_cast<double>(nbin) * nbin);   // exact: nbin is a power of two
    if (plane) {
        st = smem_opt_in(k_subfft_rows<true>, kSubSmem);
        if (st != BFS_OK) return st;
        k_subfft_rows<true><<<static_cast<unsigned>(kBlkB * nfft * nsub), 32 * kSubQ, kSubSmem, s>>>(
            z, plane, shift, t.tw, npol2, nfft, nchan, len_sft, nbin, nov_pc, mbin_adj, msamp, inv_nbin2);
        BFS_LAUNCH_CHECK("k_subfft_rows");
        return BFS_OK;
    }
    st = smem_opt_in(k_subfft_rows<false>, kSubSmem);
    if (st != BFS_OK) return st;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(kBlkB * nseg * nsub));
    cfg.blockDim = dim3(32 * kSubQ);
    cfg.dynamicSmemBytes = kSubSmem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kBlkB;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    BFS_CUDA(cudaLaunchKernelEx(&cfg, k_subfft_rows<false>, z, plane, shift, const_cast<const float2*>(t.tw), npol2, nfft,
                                nchan, len_sft, nbin, nov_pc, mbin_adj, msamp, inv_nbin2));
    BFS_LAUNCH_CHECK("k_subfft_rows");
    return BFS_OK;
}

// x (segments of kFftN complex, [pol][fft][chan]) = forward FFT of the
// unpacked int8 chunk raw; tmp holds the column-pass result (same size).
bfs_status fft_forward_guppi(const signed char* raw, float2* tmp, float2* x, long long nsamp, int noverlap,
                             int nfft, int nchan, int npol, cudaStream_t s) {
    FftTables t;
    bfs_status st = fft_tables(&t);
    if (st != BFS_OK) return st;
    BFS_ARG(nfft <= 65535 && nchan <= 65535, "too many segments or channels");
    // 16-byte copies: every group of columns starts on a word of the chunk
    const int word = 16 / npol;
    const bool vec = reinterpret_cast<uintptr_t>(raw) % 16 == 0 && nsamp % word == 0 && noverlap % word == 0;
    auto* cols = npol == 4 ? (vec ? k_fft_cols_guppi<2, true> : k_fft_cols_guppi<2, false>)
                           : (vec ? k_fft_cols_guppi<1, true> : k_fft_cols_guppi<1, false>);
    st = smem_opt_in(cols, kColSmem(npol));
    if (st != BFS_OK) return st;
    cols<<<dim3(kF / kCols, nfft, nchan), 32 * kCols, kColSmem(npol), s>>>(raw, tmp, t.twa, nsamp, noverlap, nfft,
                                                                            nchan);
    BFS_LAUNCH_CHECK("k_fft_cols_guppi");
    const long long nseg = static_cast<long long>(npol / 2) * nfft * nchan;
    BFS_ARG(nseg <= 65535, "too many segments");
    st = smem_opt_in(k_fft_rows, kRowSmem);
    if (st != BFS_OK) return st;
    k_fft_rows<<<dim3(kF / kRows, static_cast<unsigned>(nseg)), 32 * kRows, kRowSmem, s>>>(tmp, x, t.tw, t.twb);
    BFS_LAUNCH_CHECK("k_fft_rows");
    return BFS_OK;
}

}  // namespace bfs
