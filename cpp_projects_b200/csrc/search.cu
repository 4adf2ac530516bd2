// Search stage on sm_100a: per-row statistics, per-row normalisation and the
// fused normalise + boxcar + candidate-compaction kernel.
//
// Boxcar semantics (reference L/Clusterization/Clusterization.cu):
//   POW2 mode  gather_candidates_in_dynamicalArray_kernel (:420-455): for each
//              start sample t a running sum x[t] + x[t+1] + ... is tested at
//              w = 1, 2, 4, .., 2^Q; mwidth = log2 w;
//   ALL mode   do_plan_kernel / gather_candidates_in_heap_kernel (:592-671):
//              every w = 1..W, mwidth = w (the same running sum, since the
//              reference re-adds x[t..t+w-1] from x[t] in order);
//   a window is only tested when it lies inside the row; S/N = sum / sqrtf(w)
//   and a candidate is emitted when S/N > thr.
// The running sum is sequential from the start sample, as in the reference
// (a prefix-sum difference rounds differently and would flip candidates at
// the threshold).
//
// Compaction, in the canonical order (mdt, mt, width), the reference's heap
// order.  Width sets of k_boxcar_pair: a filter lists the tiles that can hold a
// candidate (low thresholds: k_boxcar_full takes them all), each tile's
// candidates are one block in that order and a scan places the blocks.  Other width sets (k_boxcar): lanes that pass a test are
// appended with one atomicAdd per warp, and the list is sorted by the key with a
// stable device radix sort.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>

#include "internal.h"
#include "search_common.cuh"

#define BFS_TRY_ST(x) do { bfs_status st_ = (x); if (st_ != BFS_OK) return st_; } while (0)

namespace bfs {
namespace {

constexpr int kBoxThreads = 256;
constexpr int kBoxTile = 1024;  // start samples per CTA
constexpr int kMaxPow2Q = 16;
constexpr int kMaxAllW = 4096;

// stats[r] = mean, stats[rows + r] = std (mode 0) or population variance (mode 1)
// launched with clusters of gridDim.x CTAs (one cluster per row)
__global__ void __launch_bounds__(kStatThreads)
k_row_stats(const float* __restrict__ plane, int rows, int cols, float* __restrict__ stats,
            int mode, int vec) {
    const int row = blockIdx.y;
    double s, q;
    cluster_row_moments(plane + static_cast<size_t>(row) * cols, row, cols, vec != 0, s, q);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const double mean = s / cols;
        double var = q / cols - mean * mean;
        if (mode == 0) {
            if (var < 0.0) var = 0.0;
            stats[row] = static_cast<float>(mean);
            stats[rows + row] = static_cast<float>(sqrt(var));
        } else {
            stats[row] = static_cast<float>(mean);
            stats[rows + row] = static_cast<float>(var);
        }
    }
}

__device__ __forceinline__ float norm_sample(float v, float m, float s) {
    return s > 0.0f ? __fdiv_rn(__fsub_rn(v, m), s) : 0.0f;
}

__global__ void k_norm_rows(const float* __restrict__ in, float* __restrict__ out, int rows,
                            int cols, const float* __restrict__ stats) {
    const int row = blockIdx.y;
    const float m = stats[row], s = stats[rows + row];
    const size_t base = static_cast<size_t>(row) * cols;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < cols; t += gridDim.x * blockDim.x)
        out[base + t] = norm_sample(__ldg(in + base + t), m, s);
}

template <int MODE>
__global__ void __launch_bounds__(kBoxThreads)
k_boxcar(const float* __restrict__ plane, int rows, int cols, const float* __restrict__ stats,
         const float* __restrict__ d_thr, float thr_host, int wmax, int snr_fast,
         bfs_cand* __restrict__ out, unsigned capacity, unsigned* __restrict__ d_count,
         int tag, int* __restrict__ tags) {
    extern __shared__ float tile[];
    const int row = blockIdx.y;
    const int t0 = blockIdx.x * kBoxTile;
    const float* x = plane + static_cast<size_t>(row) * cols;
    const int span = kBoxTile + wmax - 1;
    float m = 0.0f, sd = 0.0f;
    if (stats) { m = stats[row]; sd = stats[rows + row]; }
    for (int i = threadIdx.x; i < span; i += kBoxThreads) {
        const int t = t0 + i;
        float v = (t < cols) ? __ldg(x + t) : 0.0f;
        if (stats) v = norm_sample(v, m, sd);
        tile[i] = v;
    }
    __syncthreads();
    const float thr = d_thr ? __ldg(d_thr) : thr_host;
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int k = 0; k < kBoxTile / kBoxThreads; ++k) {
        const int i = threadIdx.x + k * kBoxThreads;
        const int t = t0 + i;
        float sum = 0.0f;
        int next = 1, pw = 0;
#pragma unroll 1
        for (int w = 1; w <= wmax; ++w) {
            const bool inside = (t + w - 1) < cols;
            if (inside) sum = __fadd_rn(sum, tile[i + w - 1]);
            bool test;
            int code;
            if (MODE == 0) {
                test = (w == next);
                code = pw;
                if (test) { next <<= 1; ++pw; }
                if (!test) continue;  // warp-uniform: w and next are the same in every lane
            } else {
                test = true;
                code = w;
            }
            const float rw = __fsqrt_rn(static_cast<float>(w));
            const float snr = snr_fast ? __fdividef(sum, rw) : __fdiv_rn(sum, rw);
            const bool pass = inside && test && (snr > thr);
            const unsigned ballot = __ballot_sync(0xffffffffu, pass);
            if (ballot) {
                const int leader = __ffs(ballot) - 1;
                unsigned base = 0;
                if (lane == leader) base = atomicAdd(d_count, static_cast<unsigned>(__popc(ballot)));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (pass) {
                    const unsigned idx = base + __popc(ballot & ((1u << lane) - 1u));
                    if (idx < capacity) {
                        bfs_cand c;
                        c.mt = t; c.mdt = row; c.mwidth = code; c.msnr = snr;
                        out[idx] = c;
                        if (tags) tags[idx] = tag;
                    }
                }
            }
        }
    }
}

// Widest window of the compile-time width sets (pow2 up to 128, every width
// up to 8) and sqrtf(w) for them, computed on the host (IEEE there too).
constexpr int kRegMaxW = 128;

struct WidthConsts {
    float sq[kRegMaxW + 1];  // sqrtf(w), w = 1..kRegMaxW (index w)
    // per filter class (window_class): 0.9999 sqrt(w) of its smallest width
    // in the set, +inf when it holds none
    float cls[8];
    float lo, hi;            // thresholds in (lo, hi]: no filter (k_boxcar_full)
    __host__ __device__ bool full(float thr) const { return thr > lo && thr <= hi; }
};

// ---- filter ---------------------------------------------------------------
// Most tiles hold no window near the threshold, so a light kernel first finds
// those that may.  With thr > 0 a window's S/N cannot pass while the sum of
// its samples' positive parts is at most thr sqrt(w): the sequential sum is at
// most the sequential sum of the positive parts (rounding is monotone), which
// rounds up by at most 128 2^-24; the normalisation, the quotient and the sums
// below add a few 2^-24, and 0.9999 covers all of it.  The positive parts are
// those of v - mean, compared with std times the bound, so the filter needs no
// division.  A window lies inside
//   class 0 (w = 1) one sample, 1 (w = 2) two samples: the tile's largest;
//   classes 2..7 (w <= 5, 9, 17, 33, 65, 129) 2, 3, 5, 9, 17, 33 neighbouring
//   blocks of 4 samples, the 16-byte pieces the row is loaded in.
// First the tile's largest block of 4 (twice, three times) and of 16 samples
// (twice, three times) are compared with the bounds, which noise rarely
// exceeds at 7 sqrt(w); only then the sums of neighbouring blocks.  NaNs count
// as 0 (a window that holds one never passes), infinities exceed every bound.
inline int window_class(int w) {
    return w == 1 ? 0 : w == 2 ? 1 : w <= 5 ? 2 : w <= 9 ? 3 : w <= 17 ? 4 : w <= 33 ? 5 : w <= 65 ? 6 : 7;
}
// Per class the largest of its sums over a tile's pair of rows, in deviations,
// that three in ten tiles of unit noise exceed.  A threshold whose bound lies
// below it for a class of the set lists more tiles than the filter saves: a
// listed tile costs three to four times one of k_boxcar_full, which then
// searches the plane unfiltered.
constexpr float kNoiseTop[8] = {3.25f, 6.5f, 8.75f, 11.2f, 15.7f, 23.8f, 38.5f, 65.5f};

// ---- ordered boxcar over row pairs -------------------------------------------
// The exact search of the tiles the filter lists, writing the candidates of
// every tile as one block in canonical order.  A CTA takes tiles of
// kPairTile consecutive starts of rows 2y and 2y + 1 from the list and stages
// them (with the WMAX - 1 samples after them) interleaved in shared memory:
// position p holds {row 2y, row 2y + 1} at sample tw + p, normalised, so one
// packed add.rn.f32x2 advances the running sums of both rows at one start —
// each half is rounded as one __fadd_rn, so the sums are the reference's
// sequential sums bit for bit.  Per width a warp first asks whether any of
// its sums exceeds the width's lower bound of passing sums; only then are
// exact quotients evaluated.  A lane's passing windows (start j, width code
// c) are bits 8 j + c, which orders them by (start, width); a scan of the
// counts over the CTA and one atomicAdd give the tile its block (row 2y's
// candidates, then row 2y + 1's).  Listed tiles are the crowded ones: two
// starts per lane keep a tile's chain of quotients and stores short (eight
// per lane and a warp per tile: 45 us at 0.3 M candidates, 13 us now).
// Record (row, tile i) = {first index, count} of row `row`'s block in tile i
// (index row * ceil(cols / kPairTile) + i), so a scan of the counts in record
// order gives every candidate its canonical position (compact_ordered).
constexpr int kPairStarts = 2;                            // starts per lane
constexpr int kPairWarps = 4;
constexpr int kPairThreads = 32 * kPairWarps;
constexpr int kPairWarpTile = 32 * kPairStarts;           // starts per warp
constexpr int kPairTile = kPairWarps * kPairWarpTile;     // starts per tile (256)

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// both halves rounded to nearest, each exactly as __fadd_rn
__device__ __forceinline__ unsigned long long add2_rn(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The width loop of one lane: kPairStarts starts from tb in both rows (win4
// = the staged tile: float4 f holds positions 2f and 2f + 1 of both rows, f0
// = the lane's first).  pass[r] gets bit 8 j + c for every passing window
// (start j, width code c) of row r, and snr[r][8 j + c] its S/N.  edge: some
// window may leave the row (tested per window).
template <int MODE, int WMAX>
__device__ __forceinline__ void pair_widths(const float4* __restrict__ win4, int f0, int tb, int cols, bool edge,
                                            float thr, float thr_lo, int snr_fast, const WidthConsts& wc,
                                            unsigned (&pass)[2], float (&snr)[2][8 * kPairStarts]) {
    constexpr int S = kPairStarts;
    constexpr int kPos = S + WMAX - 1;   // positions this lane reads
    constexpr int kVec = (kPos + 1) / 2; // float4s (two positions each)
    constexpr int kAhead = 6;            // window pairs are read this many steps before use
    unsigned long long win[2 * kVec];
    unsigned long long sum[S];
    constexpr int kPre = (S + kAhead + 1) / 2 < kVec ? (S + kAhead + 1) / 2 : kVec;
#pragma unroll
    for (int v = 0; v < kPre; ++v) {
        const float4 q = win4[f0 + v];
        win[2 * v] = pack2(q.x, q.y);
        win[2 * v + 1] = pack2(q.z, q.w);
    }
#pragma unroll
    for (int j = 0; j < S; ++j) sum[j] = 0ull;   // +0.0 in both halves
    int code = -1;
#pragma unroll
    for (int w = 1; w <= WMAX; ++w) {
        // step w reads positions w - 1 .. w + S - 2; the pair starting at
        // position w + S - 2 + kAhead is fetched now, kAhead steps early
        const int pn = w + S - 2 + kAhead;
        if ((pn & 1) == 0 && pn / 2 >= kPre && pn / 2 < kVec) {
            const float4 q = win4[f0 + pn / 2];
            win[pn] = pack2(q.x, q.y);
            win[pn + 1] = pack2(q.z, q.w);
        }
#pragma unroll
        for (int j = 0; j < S; ++j) sum[j] = add2_rn(sum[j], win[j + w - 1]);
        if (MODE == 0 && (w & (w - 1)) != 0) continue;
        ++code;   // log2 w, or w - 1
        const float sq = wc.sq[w];
        // RN(sum / sq) > thr needs sum > RN(RN(thr sq) (1 - 1e-5)) for thr > 0
        const float lim = thr_lo > -INFINITY ? __fmul_rn(__fmul_rn(thr, sq), 0.99999f) : -INFINITY;
        float h[S][2], mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < S; ++j) {
            unpack2(sum[j], h[j][0], h[j][1]);
            mx = max3f(mx, h[j][0], h[j][1]);
        }
        if (!__any_sync(0xffffffffu, mx > lim)) continue;
        // windows inside the row: starts j < inside
        const int inside = edge ? cols - (tb + w - 1) : S;
#pragma unroll
        for (int j = 0; j < S; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (!(h[j][r] > lim) || j >= inside) continue;
                const float q = snr_fast ? __fdividef(h[j][r], sq) : __fdiv_rn(h[j][r], sq);
                if (q > thr) {
                    pass[r] |= 1u << (8 * j + code);
                    snr[r][8 * j + code] = q;
                }
            }
    }
}

template <int MODE, int WMAX>
__global__ void __launch_bounds__(kPairThreads)
k_boxcar_pair(const float* __restrict__ plane, int rows, int cols, const float* __restrict__ stats,
              const float* __restrict__ d_thr, float thr_host, float thr_lo_host, int snr_fast,
              bfs_cand* __restrict__ out, unsigned capacity, unsigned* __restrict__ d_count,
              unsigned* __restrict__ rec_first, unsigned* __restrict__ rec_count,
              const unsigned* __restrict__ work, const unsigned* __restrict__ work_n, const WidthConsts wc) {
    // staged positions: every start's windows, a multiple of 4
    constexpr int kSpan = (kPairTile + WMAX - 1 + 3) / 4 * 4;
    __shared__ float4 t4[kSpan / 2 + 1];   // (a lane's last float4 may reach one past the span)
    __shared__ unsigned s_warp[2][kPairWarps], s_first;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned nwork = __ldg(work_n);
    const unsigned nwt = (cols + kPairTile - 1) / kPairTile;
    float thr = thr_host, thr_lo = thr_lo_host;
    if (d_thr) {
        thr = __ldg(d_thr);
        thr_lo = thr > 0.0f ? thr * 0.99999f : -INFINITY;
    }
#pragma unroll 1
    for (unsigned item = blockIdx.x; item < nwork; item += gridDim.x) {
        const unsigned pt = __ldg(work + item);            // row pair * nwt + tile
        const int wt = static_cast<int>(pt % nwt);
        const int tw = wt * kPairTile;
        const int row0 = 2 * static_cast<int>(pt / nwt);
        const bool has1 = row0 + 1 < rows;
        const float* x0 = plane + static_cast<size_t>(row0) * cols;
        const float* x1 = has1 ? x0 + cols : x0;
        float m0 = 0.0f, s0 = 1.0f, m1 = 0.0f, s1 = 1.0f;
        if (stats) {
            m0 = stats[row0]; s0 = stats[rows + row0];
            if (has1) { m1 = stats[row0 + 1]; s1 = stats[rows + row0 + 1]; }
        }
        __syncthreads();   // every warp is done with the tile before
        float2* t2 = reinterpret_cast<float2*>(t4);
        constexpr int kPer = (kSpan + kPairThreads - 1) / kPairThreads;
        float a[kPer], b[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int p = static_cast<int>(threadIdx.x) + kPairThreads * k;
            const bool in = p < kSpan && tw + p < cols;
            a[k] = in ? __ldg(x0 + tw + p) : 0.0f;
            b[k] = in && has1 ? __ldg(x1 + tw + p) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int p = static_cast<int>(threadIdx.x) + kPairThreads * k;
            if (p >= kSpan) continue;
            const bool in = tw + p < cols;
            t2[p] = make_float2(in && stats ? norm_sample(a[k], m0, s0) : a[k],
                                in && has1 && stats ? norm_sample(b[k], m1, s1) : b[k]);
        }
        __syncthreads();
        const int p0 = static_cast<int>(threadIdx.x) * kPairStarts;
        const int tb = tw + p0;
        unsigned pass[2] = {0u, 0u};
        float snr[2][8 * kPairStarts];   // S/N of the passing windows (indexed like their bits)
        pair_widths<MODE, WMAX>(t4, p0 / 2, tb, cols, tw + kSpan > cols, thr, thr_lo, snr_fast, wc, pass, snr);
        if (!has1) pass[1] = 0u;

        // the tile's block: row 0's candidates, then row 1's, threads in order
        const unsigned c0 = __popc(pass[0]), c1 = __popc(pass[1]);
        unsigned i01 = c0 | c1 << 16;   // inclusive scans over the lanes (at most 32 * 16 each)
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, i01, d);
            if (lane >= d) i01 += u;
        }
        if (lane == 31) { s_warp[0][warp] = i01 & 0xffffu; s_warp[1][warp] = i01 >> 16; }
        __syncthreads();
        unsigned before[2] = {0u, 0u}, tot[2] = {0u, 0u};
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int w = 0; w < kPairWarps; ++w) {
                if (w < warp) before[r] += s_warp[r][w];
                tot[r] += s_warp[r][w];
            }
        if (tot[0] + tot[1] == 0) continue;   // CTA-uniform; its records are zero already
        if (threadIdx.x == 0) {
            const unsigned first = atomicAdd(d_count, tot[0] + tot[1]);
            const size_t rec = static_cast<size_t>(row0) * nwt + wt;
            rec_first[rec] = first;
            rec_count[rec] = tot[0];
            if (has1) {
                rec_first[rec + nwt] = first + tot[0];
                rec_count[rec + nwt] = tot[1];
            }
            s_first = first;
        }
        __syncthreads();
        unsigned idx[2] = {s_first + before[0] + (i01 & 0xffffu) - c0, s_first + tot[0] + before[1] + (i01 >> 16) - c1};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (!pass[r]) continue;
#pragma unroll
            for (int bit = 0; bit < 8 * kPairStarts; ++bit) {   // bit order = (start, width) order
                if (!(pass[r] >> bit & 1u)) continue;
                if (idx[r] < capacity) {
                    bfs_cand c;
                    c.mt = tb + (bit >> 3); c.mdt = row0 + r; c.mwidth = MODE == 1 ? (bit & 7) + 1 : (bit & 7);
                    c.msnr = snr[r][bit];
                    out[idx[r]] = c;
                }
                ++idx[r];
            }
        }
    }
}

// ---- unfiltered planes: a tile per warp, eight starts per lane -----------------
// For thresholds that noise comes near in many tiles.  Bound by the
// instructions per tile, of which eight starts per lane take a third of
// k_boxcar_pair's; each warp stages its tile in its own padded shared region
// and waits for no other.  4096 x 45001 of noise, the whole call: widths 1..32
// at 4.5 deviations 454 us (918 through the filter), at 3.5 546 (1715), widths
// 1..128 at 5.0 1017 (2471); at 7.0 the filter's 169 and 294 against 432 and
// 1001 unfiltered.
// Down to a threshold of about one few of a lane's windows pass; below it
// their quotients are a chain, unless the set has one or two widths.
constexpr int kFullStarts = 8;
constexpr float kFullLow = 1.0f;
constexpr int kFullFrom = 2000;   // tiles of row pairs: fewer do not fill the chip with a warp each

// Shared layout of a warp's staged tile: logical float4 f (positions 2f,
// 2f + 1 of both rows) sits at f + f / 4, one float4 of padding after every
// four, so the eight lanes of a quarter warp — whose windows start 4 float4s
// apart — read eight different bank groups.
__device__ __forceinline__ int pad4(int f) { return f + (f >> 2); }

// pair_widths over kFullStarts starts (f0 = the lane's first logical float4;
// snr[64 r + 8 j + c] = the S/N of row r's window (start j, width code c)).
template <int MODE, int WMAX>
__device__ __forceinline__ void full_widths(const float4* __restrict__ win4, int f0, int tb, int cols, bool edge,
                                            float thr, float thr_lo, int snr_fast, const WidthConsts& wc,
                                            unsigned long long (&pass)[2], float (&snr)[128]) {
    constexpr int S = kFullStarts;
    constexpr int kPos = S + WMAX - 1;   // positions this lane reads
    constexpr int kVec = (kPos + 1) / 2; // float4s (two positions each)
    constexpr int kFullAhead = 4;            // window pairs are read this many steps before use
    unsigned long long win[2 * kVec];
    unsigned long long sum[S];
    constexpr int kPre = (S + kFullAhead + 1) / 2 < kVec ? (S + kFullAhead + 1) / 2 : kVec;
#pragma unroll
    for (int v = 0; v < kPre; ++v) {
        const float4 q = win4[pad4(f0 + v)];
        win[2 * v] = pack2(q.x, q.y);
        win[2 * v + 1] = pack2(q.z, q.w);
    }
#pragma unroll
    for (int j = 0; j < S; ++j) sum[j] = 0ull;   // +0.0 in both halves
#pragma unroll
    for (int w = 1; w <= WMAX; ++w) {
        // step w reads positions w - 1 .. w + S - 2; the pair starting at
        // position w + S - 2 + kFullAhead is fetched now, kFullAhead steps early
        const int pn = w + S - 2 + kFullAhead;
        if ((pn & 1) == 0 && pn / 2 >= kPre && pn / 2 < kVec) {
            const float4 q = win4[pad4(f0 + pn / 2)];
            win[pn] = pack2(q.x, q.y);
            win[pn + 1] = pack2(q.z, q.w);
        }
#pragma unroll
        for (int j = 0; j < S; ++j) sum[j] = add2_rn(sum[j], win[j + w - 1]);
        if (MODE == 0 && (w & (w - 1)) != 0) continue;
        const float sq = wc.sq[w];
        // RN(sum / sq) > thr needs sum > RN(RN(thr sq) (1 - 1e-5)) for thr > 0
        const float lim = thr_lo > -INFINITY ? __fmul_rn(__fmul_rn(thr, sq), 0.99999f) : -INFINITY;
        float h[2 * S], hm[S];
#pragma unroll
        for (int j = 0; j < S; ++j) {
            unpack2(sum[j], h[2 * j], h[2 * j + 1]);
            hm[j] = fmaxf(h[2 * j], h[2 * j + 1]);   // both rows at start j
        }
        float mx = max3f(hm[0], hm[1], hm[2]);
#pragma unroll
        for (int k = 3; k + 1 < S; k += 2) mx = max3f(mx, hm[k], hm[k + 1]);
        if (S % 2 == 0) mx = fmaxf(mx, hm[S - 1]);
        if (!__any_sync(0xffffffffu, mx > lim)) continue;
        const int code = (MODE == 1) ? w - 1 : 31 - __clz(w);
        // windows inside the row: starts j < inside
        const int inside = edge ? cols - (tb + w - 1) : S;
        // windows over the bound: a bit each (one code path for all of them)
        unsigned over = 0;
#pragma unroll
        for (int k = 0; k < 2 * S; ++k)
            if (h[k] > lim && (k >> 1) < inside) over |= 1u << k;
#pragma unroll 1
        while (over) {
            const int k = __ffs(over) - 1;
            over &= over - 1;
            float sj = h[0];
#pragma unroll
            for (int i = 1; i < 2 * S; ++i)
                if (i == k) sj = h[i];
            const float q = snr_fast ? __fdividef(sj, sq) : __fdiv_rn(sj, sq);
            if (q > thr) {
                const int r = k & 1, bit = 8 * (k >> 1) + code;
                pass[r] |= 1ull << bit;
                snr[64 * r + bit] = q;
            }
        }
    }
}

template <int MODE, int WMAX>
__global__ void __launch_bounds__(kPairThreads, WMAX <= 8 ? 8 : WMAX <= 32 ? 6 : WMAX <= 64 ? 4 : 2)
k_boxcar_full(const float* __restrict__ plane, int rows, int cols, const float* __restrict__ stats,
              const float* __restrict__ d_thr, float thr_host, float thr_lo_host, int snr_fast, int vec,
              bfs_cand* __restrict__ out, unsigned capacity, unsigned* __restrict__ d_count,
              unsigned* __restrict__ rec_first, unsigned* __restrict__ rec_count, const WidthConsts wc) {
    // staged positions of a warp: every start's windows, a multiple of 4
    constexpr int kSpan = (kPairTile + WMAX - 1 + 3) / 4 * 4;
    constexpr int kF4 = kSpan / 2;                      // logical float4s (kSpan positions x 2 rows)
    __shared__ float4 tile4[kPairWarps][kF4 + kF4 / 4]; // padded (pad4)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wt = blockIdx.x * kPairWarps + warp;     // warp tile
    const int tw = wt * kPairTile;
    if (tw >= cols) return;                            // warp-uniform; no other warp is waited for
    const int row0 = 2 * static_cast<int>(blockIdx.y);
    const bool has1 = row0 + 1 < rows;
    const float* x0 = plane + static_cast<size_t>(row0) * cols;
    const float* x1 = has1 ? x0 + cols : x0;
    float m0 = 0.0f, s0 = 1.0f, m1 = 0.0f, s1 = 1.0f;
    if (stats) {
        m0 = stats[row0]; s0 = stats[rows + row0];
        if (has1) { m1 = stats[row0 + 1]; s1 = stats[rows + row0 + 1]; }
    }
    auto nz = [&](float v, float m, float s) { return stats ? norm_sample(v, m, s) : v; };
    float4* t4 = tile4[warp];
    float* tile = reinterpret_cast<float*>(t4);        // position p, row r at 4 pad4(p / 2) + 2 (p % 2) + r
    const bool interior = tw + kSpan <= cols;
    if (interior && vec) {
        // 16-byte loads of both rows, every load in flight before the first use
        constexpr int kQ = kSpan / 4;                   // float4s per row
        constexpr int kPer = (kQ + 31) / 32;
        float4 a[kPer], b[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int q = lane + 32 * k;
            if (k < kPer - 1 || q < kQ) {
                a[k] = __ldg(reinterpret_cast<const float4*>(x0 + tw) + q);
                b[k] = has1 ? __ldg(reinterpret_cast<const float4*>(x1 + tw) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int q = lane + 32 * k;
            if (k < kPer - 1 || q < kQ) {
                const float b0 = has1 ? nz(b[k].x, m1, s1) : 0.0f, b1 = has1 ? nz(b[k].y, m1, s1) : 0.0f;
                const float b2 = has1 ? nz(b[k].z, m1, s1) : 0.0f, b3 = has1 ? nz(b[k].w, m1, s1) : 0.0f;
                t4[pad4(2 * q)] = make_float4(nz(a[k].x, m0, s0), b0, nz(a[k].y, m0, s0), b1);
                t4[pad4(2 * q + 1)] = make_float4(nz(a[k].z, m0, s0), b2, nz(a[k].w, m0, s0), b3);
            }
        }
    } else if (interior) {
        // 4-byte loads (rows not 16-byte aligned), all in flight first
        constexpr int kPer = (kSpan + 31) / 32;
        float a[kPer], b[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int p = lane + 32 * k;
            if (k < kPer - 1 || p < kSpan) {
                a[k] = __ldg(x0 + tw + p);
                b[k] = has1 ? __ldg(x1 + tw + p) : 0.0f;
            }
        }
        float2* t2 = reinterpret_cast<float2*>(t4);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int p = lane + 32 * k;
            if (k < kPer - 1 || p < kSpan)
                t2[2 * pad4(p >> 1) + (p & 1)] = make_float2(nz(a[k], m0, s0), has1 ? nz(b[k], m1, s1) : 0.0f);
        }
    } else {
        for (int p = lane; p < kSpan; p += 32) {
            const int t = tw + p;
            const bool in = t < cols;
            const int e = 4 * pad4(p >> 1) + 2 * (p & 1);
            tile[e] = in ? nz(__ldg(x0 + t), m0, s0) : 0.0f;
            tile[e + 1] = (in && has1) ? nz(__ldg(x1 + t), m1, s1) : 0.0f;
        }
    }
    __syncwarp();
    float thr = thr_host, thr_lo = thr_lo_host;
    if (d_thr) {
        thr = __ldg(d_thr);
        thr_lo = thr > 0.0f ? thr * 0.99999f : -INFINITY;
    }
    const int p0 = lane * kFullStarts;
    const int tb = tw + p0;
    const int f0 = p0 / 2;
    unsigned long long pass[2] = {0ull, 0ull};
    float snr[128];   // S/N of the passing windows (indexed like their bits)
    full_widths<MODE, WMAX>(t4, f0, tb, cols, !interior, thr, thr_lo, snr_fast, wc, pass, snr);
    if (!has1) pass[1] = 0ull;

    // the warp's block: row 0's candidates, then row 1's, lanes in order
    const unsigned c0 = __popcll(pass[0]), c1 = __popcll(pass[1]);
    unsigned i0 = c0, i1 = c1;   // inclusive scans over the lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned u0 = __shfl_up_sync(0xffffffffu, i0, d), u1 = __shfl_up_sync(0xffffffffu, i1, d);
        if (lane >= d) { i0 += u0; i1 += u1; }
    }
    const unsigned tot0 = __shfl_sync(0xffffffffu, i0, 31), tot1 = __shfl_sync(0xffffffffu, i1, 31);
    unsigned first = 0;
    if (lane == 0) {
        first = (tot0 + tot1) ? atomicAdd(d_count, tot0 + tot1) : 0u;
        const int nwt = (cols + kPairTile - 1) / kPairTile;
        const size_t rec = static_cast<size_t>(row0) * nwt + wt;
        rec_first[rec] = first;
        rec_count[rec] = tot0;
        if (has1) {
            rec_first[rec + nwt] = first + tot0;
            rec_count[rec + nwt] = tot1;
        }
    }
    if (tot0 + tot1 == 0) return;   // warp-uniform
    first = __shfl_sync(0xffffffffu, first, 0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        unsigned idx = first + (r ? tot0 + i1 - c1 : i0 - c0);
        unsigned long long m = pass[r];
        while (m) {   // bit order = (start, width) order
            const int bit = __ffsll(static_cast<long long>(m)) - 1;
            m &= m - 1;
            if (idx < capacity) {
                const int code = bit & 7;
                bfs_cand c;
                c.mt = tb + (bit >> 3); c.mdt = row0 + r; c.mwidth = MODE == 1 ? code + 1 : code;
                c.msnr = snr[64 * r + bit];
                out[idx] = c;
            }
            ++idx;
        }
    }
}

// b[k] -> sums j blocks further on (block index lane + 32 k + j)
template <int K>
__device__ __forceinline__ void block_shift(float (&o)[K], const float (&b)[K], int j, int lane) {
    float v[K + 1];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = __shfl_sync(0xffffffffu, b[k], (lane + j) & 31);
    v[K] = 0.0f;
#pragma unroll
    for (int k = 0; k < K; ++k) o[k] = lane + j < 32 ? v[k] : v[k + 1];
}

__device__ __forceinline__ float warp_top(float v) {   // largest of non-negative floats
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}

// Whether some window of a row may pass (warp-uniform), from its blocks'
// samples q and their mean; bound = thr std.
template <int WMAX, int K>
__device__ __forceinline__ bool row_may_pass(const float4 (&q)[K], float m, float bound, const WidthConsts& wc, int lane) {
    float b[K], big = 0.0f, b4 = 0.0f, b16 = 0.0f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const float x = fmaxf(__fsub_rn(q[k].x, m), 0.0f), y = fmaxf(__fsub_rn(q[k].y, m), 0.0f);
        const float z = fmaxf(__fsub_rn(q[k].z, m), 0.0f), w = fmaxf(__fsub_rn(q[k].w, m), 0.0f);
        b[k] = (x + y) + (z + w);
        big = fmaxf(big, fmaxf(max3f(x, y, z), w));
        if constexpr (WMAX >= 3) b4 = fmaxf(b4, b[k]);
        if constexpr (WMAX >= 16) {
            float s = b[k] + __shfl_xor_sync(0xffffffffu, b[k], 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            b16 = fmaxf(b16, s);
        }
    }
    big = warp_top(big);
    if (big > bound * wc.cls[0]) return true;
    if constexpr (WMAX >= 2)
        if (2.0f * big > bound * wc.cls[1]) return true;
    if constexpr (WMAX >= 3) {
        b4 = warp_top(b4);
        bool near = 2.0f * b4 > bound * wc.cls[2];
        if constexpr (WMAX >= 6) near |= 3.0f * b4 > bound * wc.cls[3];
        if constexpr (WMAX >= 16) {
            b16 = warp_top(b16);
            near |= 2.0f * b16 > bound * wc.cls[4];
            if constexpr (WMAX >= 32) near |= 3.0f * b16 > bound * wc.cls[5];
            if constexpr (WMAX >= 64) near |= 5.0f * b16 > bound * wc.cls[6];
            if constexpr (WMAX >= 128) near |= 9.0f * b16 > bound * wc.cls[7];
        }
        if (!near) return false;
        bool over = false;
        float sum[K], t[K];   // sums of 2, 4, 8, .. blocks
        auto test = [&](int cls) {
#pragma unroll
            for (int k = 0; k < K; ++k) over |= t[k] > bound * wc.cls[cls];
        };
        auto plus = [&](const float (&x)[K], int j) {   // t = sum + x shifted
            block_shift<K>(t, x, j, lane);
#pragma unroll
            for (int k = 0; k < K; ++k) t[k] += sum[k];
        };
        auto keep = [&]() {
#pragma unroll
            for (int k = 0; k < K; ++k) sum[k] = t[k];
        };
#pragma unroll
        for (int k = 0; k < K; ++k) sum[k] = b[k];
        plus(b, 1);
        test(2);
        if constexpr (WMAX >= 6) {
            keep();
            plus(b, 2);
            test(3);
        }
        if constexpr (WMAX >= 16) {
            plus(sum, 2);
            keep();
            plus(b, 4);
            test(4);
        }
        if constexpr (WMAX >= 32) {
            plus(sum, 4);
            keep();
            plus(b, 8);
            test(5);
        }
        if constexpr (WMAX >= 64) {
            plus(sum, 8);
            keep();
            plus(b, 16);
            test(6);
        }
        if constexpr (WMAX >= 128) {
            plus(sum, 16);
            keep();
#pragma unroll
            for (int k = 0; k < K; ++k) t[k] = sum[k] + (k + 1 < K ? b[k + 1] : 0.0f);   // 32 blocks further on
            test(7);
        }
        return __any_sync(0xffffffffu, over);
    }
    return false;
}

// One warp per (row pair, warp tile): its records zeroed, and the tile put on
// the work list when a window of one of its rows may pass (all of them with
// thr <= 0).  Rows are read in 16-byte pieces of memory: where a row's samples
// tw.. start `ph` floats into a piece, the samples before tw in it only raise
// the sums.  Pieces that leave the row are read sample by sample, the mean
// taken for what lies outside.  HBM-bound: 4096 x 45001 in 141 us (5.2 TB/s)
// with 56 warps per SM, 178 us with 40; the whole search of that plane took
// 330 us in one kernel, of a 512 x 32768 plane with 0.3 M candidates 89 us,
// now 14.5 + 13 us.
constexpr int kFilterThreads = 128;
template <int WMAX>
__global__ void __launch_bounds__(kFilterThreads, WMAX <= 32 ? 14 : 10)
k_boxcar_filter(const float* __restrict__ plane, int rows, int cols, const float* __restrict__ stats,
                const float* __restrict__ d_thr, float thr_host, unsigned* __restrict__ rec_count,
                unsigned* __restrict__ work, unsigned* __restrict__ work_n, const WidthConsts wc) {
    constexpr int kSpan = (kPairTile + WMAX - 1 + 3) / 4 * 4;
    constexpr int kBlocks = kSpan / 4 + 1;
    constexpr int kPer = (kBlocks + 31) / 32;
    const unsigned nwt = (cols + kPairTile - 1) / kPairTile;
    const unsigned wt = blockIdx.x * (kFilterThreads / 32) + (threadIdx.x >> 5);
    if (wt >= nwt) return;   // warp-uniform
    const int lane = threadIdx.x & 31, tw = static_cast<int>(wt) * kPairTile;
    const unsigned pt = blockIdx.y * nwt + wt;
    const int row0 = 2 * static_cast<int>(blockIdx.y);
    const float thr = d_thr ? __ldg(d_thr) : thr_host;
    if (d_thr && wc.full(thr)) {   // (known on the device only: the caller searches unfiltered)
        if (pt == 0 && lane == 0) work_n[1] = 1u;
        return;
    }
    const bool has1 = row0 + 1 < rows;
    bool may = !(thr > 0.0f);
    if (!may) {
        float4 q[2][kPer];
        float m[2] = {0.0f, 0.0f}, sd[2] = {1.0f, 1.0f};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (r && !has1) continue;
            if (stats) { m[r] = __ldg(stats + row0 + r); sd[r] = __ldg(stats + rows + row0 + r); }
            const float* x = plane + static_cast<size_t>(row0 + r) * cols;
            const int ph = static_cast<int>((reinterpret_cast<uintptr_t>(x + tw) >> 2) & 3);
            if ((tw >= 4 || ph == 0) && tw + 4 * kBlocks <= cols) {   // no piece leaves the row
#pragma unroll
                for (int k = 0; k < kPer; ++k)
                    if (k < kPer - 1 || lane + 32 * k < kBlocks)
                        q[r][k] = __ldg(reinterpret_cast<const float4*>(x + tw + 4 * (lane + 32 * k) - ph));
                    else
                        q[r][k] = make_float4(m[r], m[r], m[r], m[r]);
            } else {
#pragma unroll
                for (int k = 0; k < kPer; ++k) {
                    float f[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int t = tw + 4 * (lane + 32 * k) - ph + j;
                        f[j] = t >= tw && t < min(cols, tw + kSpan) ? __ldg(x + t) : m[r];
                    }
                    q[r][k] = make_float4(f[0], f[1], f[2], f[3]);
                }
            }
        }
        // std 0 or NaN: every sample is 0; std beyond the bounds' range: not filtered
#pragma unroll
        for (int r = 0; r < 2; ++r)
            if (!may && (r == 0 || has1) && sd[r] > 0.0f)
                may = sd[r] < 1e-30f || sd[r] > 1e30f || row_may_pass<WMAX, kPer>(q[r], m[r], thr * sd[r], wc, lane);
    }
    if (lane == 0) {
        const size_t rec = static_cast<size_t>(row0) * nwt + wt;
        rec_count[rec] = 0u;
        if (has1) rec_count[rec + nwt] = 0u;
        if (may) work[atomicAdd(work_n, 1u)] = pt;
    }
}

// Candidates of records [0, nrec) moved to their canonical positions
// (pos = exclusive scan of the counts); tags[pos..] = the record's beam when
// tags is given (beam b owns records [beam_rec[b], beam_rec[b + 1])).  A warp
// takes 32 consecutive records.
__global__ void k_compact_records(const bfs_cand* __restrict__ src, const unsigned* __restrict__ rec_first,
                                  const unsigned* __restrict__ rec_count, const unsigned* __restrict__ rec_pos,
                                  long long nrec, const long long* __restrict__ beam_rec, int nb,
                                  bfs_cand* __restrict__ dst, int* __restrict__ tags) {
    const long long r = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    unsigned n = 0, from = 0, to = 0;
    int beam = 0;
    if (r < nrec) {
        n = rec_count[r];
        if (n) {
            from = rec_first[r];
            to = rec_pos[r];
            if (tags) {   // last beam whose first record is <= r
                int lo = 0, hi = nb - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (beam_rec[mid] <= r) lo = mid; else hi = mid - 1;
                }
                beam = lo;
            }
        }
    }
    // the warp's records follow one another in dst: its lanes take the
    // candidates of all of them in turn (one record at a time left most lanes
    // idle: 16.5 us for 65536 records of ~5)
    unsigned end = n;   // inclusive scan of the counts
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += u;
    }
    const unsigned total = __shfl_sync(0xffffffffu, end, 31);
    if (total == 0) return;
    const unsigned first = from - (end - n);   // source of the warp's candidate i: first + i (of its record)
    const unsigned some = __ballot_sync(0xffffffffu, n != 0);
    const unsigned to0 = __shfl_sync(0xffffffffu, to, __ffs(some) - 1);
    for (unsigned i0 = 0; i0 < total; i0 += 32) {   // warp-uniform
        const unsigned i = i0 + lane;
        int rec = 0;   // records whose end is <= i
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const unsigned e = __shfl_sync(0xffffffffu, end, rec + d - 1);
            if (e <= i) rec += d;
        }
        const unsigned f = __shfl_sync(0xffffffffu, first, rec & 31);
        const int cb = __shfl_sync(0xffffffffu, beam, rec & 31);
        if (i < total) {
            dst[to0 + i] = src[f + i];
            if (tags) tags[to0 + i] = cb;
        }
    }
}

// Canonical key of a candidate: (row * cols + start) << wbits | width code,
// with the width code 0..Q (pow2 mode) or w-1 (all-widths mode).
__device__ __forceinline__ unsigned long long cand_key(const bfs_cand& v, int cols, int mode, int wbits) {
    const unsigned long long cell = static_cast<unsigned long long>(v.mdt) * cols + v.mt;
    const unsigned long long code = static_cast<unsigned long long>(mode == 0 ? v.mwidth : v.mwidth - 1);
    return (cell << wbits) | code;
}

__global__ void k_cand_keys(const bfs_cand* __restrict__ c, unsigned n, int cols, int mode, int wbits,
                            unsigned long long* __restrict__ keys, unsigned* __restrict__ vals) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    keys[i] = cand_key(c[i], cols, mode, wbits);
    vals[i] = i;
}

__global__ void k_gather_cands(const bfs_cand* __restrict__ src, const unsigned* __restrict__ idx,
                               unsigned n, bfs_cand* __restrict__ dst) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[idx[i]];
}

// 32-bit variant: the key holds the whole position, the S/N rides along as
// the sort value, and the records are rebuilt from (key, S/N).
__global__ void k_cand_keys32(const bfs_cand* __restrict__ c, unsigned n, int cols, int mode, int wbits,
                              unsigned* __restrict__ keys, unsigned* __restrict__ vals) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bfs_cand v = c[i];
    keys[i] = static_cast<unsigned>(cand_key(v, cols, mode, wbits));
    vals[i] = __float_as_uint(v.msnr);
}

__global__ void k_cand_decode32(const unsigned* __restrict__ keys, const unsigned* __restrict__ vals,
                                unsigned n, int cols, int mode, int wbits, bfs_cand* __restrict__ out) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned k = keys[i];
    const unsigned cell = wbits ? (k >> wbits) : k;
    const int code = static_cast<int>(k & ((1u << wbits) - 1u));
    bfs_cand c;
    c.mt = static_cast<int>(cell % static_cast<unsigned>(cols));
    c.mdt = static_cast<int>(cell / static_cast<unsigned>(cols));
    c.mwidth = mode == 0 ? code : code + 1;
    c.msnr = __uint_as_float(vals[i]);
    out[i] = c;
}

int bits_for(unsigned long long v) {
    int b = 0;
    while (b < 64 && (v >> b) != 0ull) ++b;
    return b;
}

}  // namespace

// Sorts n candidates of a rows x cols plane into the canonical order in place.
// Scratch comes from the stream-ordered pool allocator.
bfs_status sort_candidates_canonical(bfs_cand* d_c, unsigned n, int rows, int cols, int mode,
                                     int param, cudaStream_t s) {
    if (n < 2) return BFS_OK;
    const int wbits = bits_for(static_cast<unsigned long long>(mode == 0 ? param : param - 1));
    const int cell_bits = bits_for(static_cast<unsigned long long>(rows) * cols - 1);
    const int end_bit = cell_bits + wbits;
    const int th = 256, bl = static_cast<int>((n + th - 1) / th);
    void* cub_tmp = nullptr;
    size_t cub_bytes = 0;
    if (end_bit <= 32) {
        unsigned *k = nullptr, *v = nullptr;
        BFS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, k, k, v, v,
                                                 static_cast<int>(n), 0, end_bit, s));
        BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&k), n * sizeof(unsigned) * 4, s));
        v = k + 2 * static_cast<size_t>(n);
        BFS_TRY_ST(stream_alloc(&cub_tmp, cub_bytes ? cub_bytes : 16, s));
        k_cand_keys32<<<bl, th, 0, s>>>(d_c, n, cols, mode, wbits, k, v);
        BFS_LAUNCH_CHECK("k_cand_keys32");
        BFS_CUDA(cub::DeviceRadixSort::SortPairs(cub_tmp, cub_bytes, k, k + n, v, v + n,
                                                 static_cast<int>(n), 0, end_bit, s));
        k_cand_decode32<<<bl, th, 0, s>>>(k + n, v + n, n, cols, mode, wbits, d_c);
        BFS_LAUNCH_CHECK("k_cand_decode32");
        BFS_CUDA(cudaFreeAsync(k, s));
        BFS_CUDA(cudaFreeAsync(cub_tmp, s));
        return BFS_OK;
    }
    unsigned long long *k_in = nullptr, *k_out = nullptr;
    unsigned *v_in = nullptr, *v_out = nullptr;
    bfs_cand* tmp = nullptr;
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, k_in, k_out, v_in, v_out,
                                             static_cast<int>(n), 0, end_bit, s));
    BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&k_in), n * sizeof(unsigned long long) * 2, s));
    k_out = k_in + n;
    BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&v_in), n * sizeof(unsigned) * 2, s));
    v_out = v_in + n;
    BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&tmp), n * sizeof(bfs_cand), s));
    BFS_TRY_ST(stream_alloc(&cub_tmp, cub_bytes ? cub_bytes : 16, s));
    k_cand_keys<<<bl, th, 0, s>>>(d_c, n, cols, mode, wbits, k_in, v_in);
    BFS_LAUNCH_CHECK("k_cand_keys");
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(cub_tmp, cub_bytes, k_in, k_out, v_in, v_out,
                                             static_cast<int>(n), 0, end_bit, s));
    k_gather_cands<<<bl, th, 0, s>>>(d_c, v_out, n, tmp);
    BFS_LAUNCH_CHECK("k_gather_cands");
    BFS_CUDA(cudaMemcpyAsync(d_c, tmp, n * sizeof(bfs_cand), cudaMemcpyDeviceToDevice, s));
    BFS_CUDA(cudaFreeAsync(k_in, s));
    BFS_CUDA(cudaFreeAsync(v_in, s));
    BFS_CUDA(cudaFreeAsync(tmp, s));
    BFS_CUDA(cudaFreeAsync(cub_tmp, s));
    return BFS_OK;
}

namespace {
__global__ void k_tagged_keys(const bfs_cand* __restrict__ c, const int* __restrict__ tags, unsigned n,
                              int row_bits, int col_bits, int mode, int wbits,
                              unsigned long long* __restrict__ keys, unsigned* __restrict__ vals) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bfs_cand v = c[i];
    const unsigned long long code = static_cast<unsigned long long>(mode == 0 ? v.mwidth : v.mwidth - 1);
    unsigned long long k = static_cast<unsigned long long>(tags[i]);
    k = (k << row_bits) | static_cast<unsigned long long>(v.mdt);
    k = (k << col_bits) | static_cast<unsigned long long>(v.mt);
    keys[i] = (k << wbits) | code;
    vals[i] = i;
}

__global__ void k_gather_tagged(const bfs_cand* __restrict__ src, const int* __restrict__ tsrc,
                                const unsigned* __restrict__ idx, unsigned n, bfs_cand* __restrict__ dst,
                                int* __restrict__ tdst) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { dst[i] = src[idx[i]]; tdst[i] = tsrc[idx[i]]; }
}
}  // namespace

// Canonical order across beams: (tag, row, sample, width); candidates and
// their tags are permuted together (into dst / tdst).
bfs_status sort_tagged_candidates(const bfs_cand* d_c, const int* d_tags, unsigned n, int max_rows,
                                  int max_cols, int max_tag, int mode, int param, bfs_cand* d_dst,
                                  int* d_tdst, cudaStream_t s) {
    if (n == 0) return BFS_OK;
    const int wbits = bits_for(static_cast<unsigned long long>(mode == 0 ? param : param - 1));
    const int row_bits = bits_for(static_cast<unsigned long long>(max_rows - 1));
    const int col_bits = bits_for(static_cast<unsigned long long>(max_cols - 1));
    const int tag_bits = bits_for(static_cast<unsigned long long>(max_tag));
    const int end_bit = tag_bits + row_bits + col_bits + wbits;
    BFS_ARG(end_bit <= 64, "candidate key needs %d bits", end_bit);
    unsigned long long* k = nullptr;
    unsigned* v = nullptr;
    void* tmp = nullptr;
    size_t tmp_bytes = 0;
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, k, k, v, v, static_cast<int>(n), 0,
                                             end_bit > 0 ? end_bit : 1, s));
    BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&k), sizeof(unsigned long long) * 2 * n, s));
    BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&v), sizeof(unsigned) * 2 * n, s));
    BFS_TRY_ST(stream_alloc(&tmp, tmp_bytes, s));
    const int th = 256, bl = static_cast<int>((n + th - 1) / th);
    k_tagged_keys<<<bl, th, 0, s>>>(d_c, d_tags, n, row_bits, col_bits, mode, wbits, k, v);
    BFS_LAUNCH_CHECK("k_tagged_keys");
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, k, k + n, v, v + n, static_cast<int>(n), 0,
                                             end_bit > 0 ? end_bit : 1, s));
    k_gather_tagged<<<bl, th, 0, s>>>(d_c, d_tags, v + n, n, d_dst, d_tdst);
    BFS_LAUNCH_CHECK("k_gather_tagged");
    BFS_CUDA(cudaFreeAsync(k, s));
    BFS_CUDA(cudaFreeAsync(v, s));
    BFS_CUDA(cudaFreeAsync(tmp, s));
    return BFS_OK;
}

bfs_status launch_row_stats(const float* d_in, int rows, int cols, float* d_stats, int mode,
                            cudaStream_t s) {
    BFS_ARG(d_in && d_stats, "null argument");
    BFS_ARG(rows >= 1 && cols >= 1, "bad shape %dx%d", rows, cols);
    BFS_ARG(rows <= 65535, "rows > 65535 not supported");
    // CTAs per row: doubled while the grid is under two waves of 256-thread
    // CTAs (8 per SM) and every thread still reads >= 32 samples
    int dev = 0, sms = 0;
    BFS_CUDA(cudaGetDevice(&dev));
    BFS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int split = 1;
    while (split < kStatMaxCluster && static_cast<long long>(rows) * split < 16LL * sms &&
           cols / (2 * split) >= 32 * kStatThreads)
        split *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(split, rows);
    cfg.blockDim = dim3(kStatThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = split;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int vec = (reinterpret_cast<uintptr_t>(d_in) & 15) == 0 ? 1 : 0;
    BFS_CUDA(cudaLaunchKernelEx(&cfg, k_row_stats, d_in, rows, cols, d_stats, mode, vec));
    return BFS_OK;
}

bfs_status launch_boxcar(const float* d_plane, int rows, int cols, const float* d_stats,
                         float thr, const float* d_thr, int mode, int param, int snr_fast,
                         bfs_cand* d_out, unsigned capacity, unsigned* d_count, cudaStream_t s,
                         int tag, int* d_tags) {
    BFS_ARG(d_plane && d_count, "null argument");
    BFS_ARG(rows >= 1 && cols >= 1 && rows <= 65535, "bad shape %dx%d", rows, cols);
    BFS_ARG(capacity == 0 || d_out, "d_out is null");
    int wmax;
    if (mode == BFS_WIDTHS_POW2) {
        BFS_ARG(param >= 0 && param <= kMaxPow2Q, "Q must be in [0, %d]", kMaxPow2Q);
        wmax = 1 << param;
    } else if (mode == BFS_WIDTHS_ALL) {
        BFS_ARG(param >= 1 && param <= kMaxAllW, "W must be in [1, %d]", kMaxAllW);
        wmax = param;
    } else {
        return fail(BFS_ERR_ARG, "unknown widths_mode %d", mode);
    }
    dim3 grid((cols + kBoxTile - 1) / kBoxTile, rows);
    const size_t smem = sizeof(float) * (kBoxTile + wmax - 1);
    if (mode == BFS_WIDTHS_POW2) {
        if (smem > 48 * 1024)
            BFS_CUDA(cudaFuncSetAttribute(k_boxcar<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(smem)));
        k_boxcar<0><<<grid, kBoxThreads, smem, s>>>(d_plane, rows, cols, d_stats, d_thr, thr, wmax,
                                                    snr_fast, d_out, capacity, d_count, tag, d_tags);
    } else {
        if (smem > 48 * 1024)
            BFS_CUDA(cudaFuncSetAttribute(k_boxcar<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(smem)));
        k_boxcar<1><<<grid, kBoxThreads, smem, s>>>(d_plane, rows, cols, d_stats, d_thr, thr, wmax,
                                                    snr_fast, d_out, capacity, d_count, tag, d_tags);
    }
    BFS_LAUNCH_CHECK("k_boxcar");
    return BFS_OK;
}

// Whether launch_boxcar_ordered handles a width set (pow2 up to 128 or every
// width up to 8: at most 8 width codes per start).
bool boxcar_ordered_supported(int mode, int param) {
    if (mode == BFS_WIDTHS_POW2) return param >= 0 && param <= 7;
    if (mode == BFS_WIDTHS_ALL) return param >= 1 && param <= 8;
    return false;
}

long long boxcar_ordered_records(int rows, int cols) {
    return static_cast<long long>(rows) * ((cols + kPairTile - 1) / kPairTile);
}

// The boxcar with canonical per-tile output (k_boxcar_pair): candidates go to
// d_out in blocks, one per (row, warp tile), each in canonical order; records
// rec_first / rec_count (boxcar_ordered_records entries, (row, tile) order)
// locate the blocks for compact_ordered.  work: one entry per row pair and
// warp tile; *work_n: 0.  A threshold in device memory (d_thr) may ask for the
// unfiltered search: work_n[1] (0 before) is then 1, nothing was searched, and
// the call is to be made again with `full`.
bfs_status launch_boxcar_ordered(const float* d_plane, int rows, int cols, const float* d_stats, float thr,
                                 const float* d_thr, int mode, int param, int snr_fast, bfs_cand* d_out,
                                 unsigned capacity, unsigned* d_count, unsigned* rec_first, unsigned* rec_count,
                                 unsigned* work, unsigned* work_n, cudaStream_t s, bool full) {
    BFS_ARG(d_plane && d_count && rec_first && rec_count && work && work_n, "null argument");
    BFS_ARG(rows >= 1 && cols >= 1, "bad shape %dx%d", rows, cols);
    BFS_ARG((rows + 1) / 2 <= 65535, "rows > 131070 not supported");
    BFS_ARG(capacity == 0 || d_out, "d_out is null");
    BFS_ARG(boxcar_ordered_supported(mode, param), "width set (%d, %d) has no ordered kernel", mode, param);
    const float thr_lo = thr > 0.0f ? thr * 0.99999f : -INFINITY;
    WidthConsts wc;
    for (int w = 0; w <= kRegMaxW; ++w) wc.sq[w] = std::sqrt(static_cast<float>(w));  // IEEE-correct on the host
    for (float& c : wc.cls) c = INFINITY;
    const int widest = mode == BFS_WIDTHS_POW2 ? 1 << param : param;
    for (int w = 1; w <= widest; w = mode == BFS_WIDTHS_POW2 ? 2 * w : w + 1)
        wc.cls[window_class(w)] = std::min(wc.cls[window_class(w)], 0.9999f * wc.sq[w]);
    const long long pairs = boxcar_ordered_records((rows + 1) / 2, cols);
    BFS_ARG(pairs < (1ll << 31), "too many boxcar tiles (%lld)", pairs);
    constexpr int kPerCta = kFilterThreads / 32 * kPairTile;
    const dim3 fgrid((cols + kPerCta - 1) / kPerCta, (rows + 1) / 2);
    // the searching kernel's CTAs take the listed tiles in turn
    const int grid = static_cast<int>(std::min<long long>(pairs, 148LL * 8));
    const int nwidths = mode == BFS_WIDTHS_POW2 ? param + 1 : param;
    wc.lo = nwidths >= 3 ? kFullLow : 0.0f;
    wc.hi = 0.0f;
    for (int c = 0; c < 8 && pairs >= kFullFrom; ++c) wc.hi = std::max(wc.hi, kNoiseTop[c] / wc.cls[c]);
    const int vec = cols % 4 == 0 && reinterpret_cast<uintptr_t>(d_plane) % 16 == 0 ? 1 : 0;
#define BFS_BOX_PAIR(M, W)                                                                                        \
    if (full || (!d_thr && wc.full(thr))) {                                                                       \
        k_boxcar_full<M, W><<<fgrid, kPairThreads, 0, s>>>(d_plane, rows, cols, d_stats, d_thr, thr, thr_lo,      \
                                                           snr_fast, vec, d_out, capacity, d_count, rec_first,    \
                                                           rec_count, wc);                                        \
        break;                                                                                                    \
    }                                                                                                             \
    k_boxcar_filter<W><<<fgrid, kFilterThreads, 0, s>>>(d_plane, rows, cols, d_stats, d_thr, thr, rec_count,     \
                                                        work, work_n, wc);                                        \
    k_boxcar_pair<M, W><<<grid, kPairThreads, 0, s>>>(d_plane, rows, cols, d_stats, d_thr, thr, thr_lo, snr_fast,  \
                                                      d_out, capacity, d_count, rec_first, rec_count, work,        \
                                                      work_n, wc)
    if (mode == BFS_WIDTHS_POW2) {
        switch (param) {
            case 0: BFS_BOX_PAIR(0, 1); break;
            case 1: BFS_BOX_PAIR(0, 2); break;
            case 2: BFS_BOX_PAIR(0, 4); break;
            case 3: BFS_BOX_PAIR(0, 8); break;
            case 4: BFS_BOX_PAIR(0, 16); break;
            case 5: BFS_BOX_PAIR(0, 32); break;
            case 6: BFS_BOX_PAIR(0, 64); break;
            default: BFS_BOX_PAIR(0, 128); break;
        }
    } else {
        switch (param) {
            case 1: BFS_BOX_PAIR(1, 1); break;
            case 2: BFS_BOX_PAIR(1, 2); break;
            case 3: BFS_BOX_PAIR(1, 3); break;
            case 4: BFS_BOX_PAIR(1, 4); break;
            case 5: BFS_BOX_PAIR(1, 5); break;
            case 6: BFS_BOX_PAIR(1, 6); break;
            case 7: BFS_BOX_PAIR(1, 7); break;
            default: BFS_BOX_PAIR(1, 8); break;
        }
    }
#undef BFS_BOX_PAIR
    BFS_LAUNCH_CHECK("k_boxcar_pair");
    return BFS_OK;
}

// The candidates of nrec records (blocks in src written by
// launch_boxcar_ordered, every count summing to at most the capacity src was
// written with) in canonical order in dst; tags (optional) = each candidate's
// beam, beam b owning records [beam_rec[b], beam_rec[b + 1]) (beam_rec on the
// device, nb + 1 entries).  Scratch from the stream-ordered pool.
bfs_status compact_ordered(const bfs_cand* src, const unsigned* rec_first, const unsigned* rec_count,
                           long long nrec, const long long* beam_rec, int nb, bfs_cand* dst, int* tags,
                           cudaStream_t s) {
    if (nrec <= 0) return BFS_OK;
    BFS_ARG(nrec < (1ll << 31), "too many boxcar tiles (%lld)", nrec);
    BFS_ARG(!tags || (beam_rec && nb >= 1), "tags need the beams' record offsets");
    const int th = 256;
    const long long blocks = (nrec + th - 1) / th;
    BFS_ARG(blocks < (1ll << 31), "too many boxcar tiles (%lld)", nrec);
    unsigned* pos = nullptr;
    size_t tmp_bytes = 0;
    BFS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, rec_count, pos, static_cast<int>(nrec), s));
    const size_t pos_bytes = (sizeof(unsigned) * nrec + 255) & ~static_cast<size_t>(255);
    bfs_status st = stream_alloc(reinterpret_cast<void**>(&pos), pos_bytes + tmp_bytes, s);
    void* tmp = reinterpret_cast<char*>(pos) + pos_bytes;
    if (st == BFS_OK) {
        cudaError_t e = cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, rec_count, pos, static_cast<int>(nrec), s);
        if (e == cudaSuccess) {
            k_compact_records<<<static_cast<unsigned>(blocks), th, 0, s>>>(src, rec_first, rec_count, pos, nrec,
                                                                            beam_rec, nb, dst, tags);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) st = fail(BFS_ERR_CUDA, "candidate compaction: %s", cudaGetErrorString(e));
    }
    if (pos) cudaFreeAsync(pos, s);
    return st;
}

}  // namespace bfs

using namespace bfs;

extern "C" bfs_status bfs_row_stats(const float* d_in, int rows, int cols, float* d_stats,
                                    void* stream) {
    return launch_row_stats(d_in, rows, cols, d_stats, 0, as_stream(stream));
}

extern "C" bfs_status bfs_norm_rows(const float* d_in, float* d_out, int rows, int cols,
                                    float* d_stats, void* stream) {
    BFS_ARG(d_in && d_out, "null argument");
    BFS_ARG(rows >= 1 && cols >= 1 && rows <= 65535, "bad shape %dx%d", rows, cols);
    cudaStream_t s = as_stream(stream);
    float* stats = d_stats;
    if (!stats) BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&stats), sizeof(float) * 2 * rows, s));
    bfs_status st = launch_row_stats(d_in, rows, cols, stats, 0, s);
    if (st == BFS_OK) {
        dim3 grid(std::min((cols + 255) / 256, 64), rows);
        k_norm_rows<<<grid, 256, 0, s>>>(d_in, d_out, rows, cols, stats);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) st = fail(BFS_ERR_CUDA, "k_norm_rows: %s", cudaGetErrorString(e));
    }
    if (!d_stats) cudaFreeAsync(stats, s);
    return st;
}

extern "C" bfs_status bfs_boxcar_gather(const float* d_plane, int rows, int cols,
                                        const float* d_stats, float thr, const float* d_thr,
                                        int widths_mode, int param, int snr_fast, bfs_cand* d_out,
                                        uint32_t capacity, uint32_t* h_count, void* stream) {
    BFS_ARG(h_count != nullptr, "h_count is null");
    BFS_ARG(d_plane != nullptr, "null argument");
    BFS_ARG(rows >= 1 && cols >= 1 && rows <= 65535, "bad shape %dx%d", rows, cols);
    cudaStream_t s = as_stream(stream);
    // width sets with an ordered kernel: candidates come out in per-tile
    // canonical blocks, then one scan + move puts them in canonical order;
    // others: atomic appends, then a radix sort by the canonical key
    const bool ordered = boxcar_ordered_supported(widths_mode, param);
    const long long nrec = ordered ? boxcar_ordered_records(rows, cols) : 0;
    // one piece: candidate and work-list counts, first[nrec], count[nrec], work[nrec]
    unsigned* d_count = nullptr;
    BFS_TRY_ST(stream_alloc(reinterpret_cast<void**>(&d_count), sizeof(unsigned) * (64 + 3 * nrec), s));
    unsigned* rec = d_count + 64;
    bfs_status st = BFS_OK;
    {
        cudaError_t e = cudaMemsetAsync(d_count, 0, 3 * sizeof(unsigned), s);
        if (e != cudaSuccess) st = fail(BFS_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    }
    auto search = [&](bool full) {
        return ordered ? launch_boxcar_ordered(d_plane, rows, cols, d_stats, thr, d_thr, widths_mode, param, snr_fast,
                                               d_out, capacity, d_count, rec, rec + nrec, rec + 2 * nrec, d_count + 1, s,
                                               full)
                       : launch_boxcar(d_plane, rows, cols, d_stats, thr, d_thr, widths_mode, param,
                                       snr_fast, d_out, capacity, d_count, s, 0, nullptr);
    };
    if (st == BFS_OK) st = search(false);
    unsigned words[3] = {0, 0, 0};
    if (st == BFS_OK) st = read_back(words, d_count, 3, s);
    if (st == BFS_OK && words[2]) {
        st = search(true);
        if (st == BFS_OK) st = read_back(words, d_count, 1, s);
    }
    const unsigned count = words[0];
    if (st == BFS_OK) {
        *h_count = count;
        const unsigned n = count < capacity ? count : capacity;
        if (ordered && count <= capacity && count >= 2) {
            bfs_cand* tmp = nullptr;
            st = stream_alloc(reinterpret_cast<void**>(&tmp), sizeof(bfs_cand) * count, s);
            if (st == BFS_OK) st = compact_ordered(d_out, rec, rec + nrec, nrec, nullptr, 0, tmp, nullptr, s);
            if (st == BFS_OK) {
                cudaError_t e = cudaMemcpyAsync(d_out, tmp, sizeof(bfs_cand) * count, cudaMemcpyDeviceToDevice, s);
                if (e != cudaSuccess) st = fail(BFS_ERR_CUDA, "cudaMemcpyAsync: %s", cudaGetErrorString(e));
            }
            if (tmp) cudaFreeAsync(tmp, s);
        } else if (!ordered || count > capacity) {
            // (ordered overflow: the blocks that fit, sorted)
            st = sort_candidates_canonical(d_out, n, rows, cols, widths_mode, param, s);
        }
    }
    cudaFreeAsync(d_count, s);
    if (st != BFS_OK) return st;
    if (count > capacity)
        return fail(BFS_ERR_OVERFLOW, "%u candidates found, capacity %u", count, capacity);
    return BFS_OK;
}
