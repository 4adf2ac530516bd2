// Adjoint FDMT and adjoint boxcar S/N on sm_100a (no reference counterpart:
// the reference has no gradients).  They make the search differentiable, so
// per-channel weights (bandpass / RFI masks) can be optimised against the
// S/N of detections.
//
// Every FDMT level is linear in its input plane, so the adjoint needs only
// the incoming gradient, never the forward planes: nothing is stored and
// nothing is recomputed beyond one pass per level, in two ping-pong planes
// like the forward.
//
//   merge level l   forward  out[g][t] = in[a_g][t] + [t >= s_g] in[b_g][t - s_g]
//                   adjoint  gin[i][u] = sum over the level-l rows g that read
//                            row i of gout[g][u + s] (s = 0 as tail a_g, s_g as
//                            head b_g; terms with u + s >= ncols vanish) — a
//                            gather over the plan's inverse row tables, summed
//                            in ascending g, so the FP32 result is fixed;
//   level 0         forward  P[c,r][t] = [t >= r] mean(x[c][t-r .. t])
//                   adjoint  gx[c][u] = sum_{r'} RN(1/(r'+1)) *
//                            sum_{r=0..r'} [u+r >= r'][u+r < ncols] g0[c,r'][u+r]
//                            (inner sums r ascending, outer r' ascending).
//
// Boxcar S/N at a cell (row d, start t, width w) of the plane y with row mean
// m_d and standard deviation s_d (population, as bfs_row_stats gives):
//   S = sum_{j<w} z(y[d][t+j]) / sqrt(w),  z(v) = (v - m_d) / s_d,
// evaluated exactly as the boxcar kernels do.  Its gradient, with m_d and s_d
// functions of the row (N = ncols samples):
//   dS/dy[d][u] = ([t <= u < t+w] - w/N) / (s_d sqrt(w)) - S (y[d][u] - m_d) / (N s_d^2).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>

#include "fdmt_plan.h"
#include "internal.h"
#include "row_ops.cuh"

namespace bfs {
namespace {

constexpr int kAdjThreads = 128;   // measured: 128 > 256 > 512 on 1024 x 65536
constexpr int kAdjVecs = 2;       // float4 column groups per thread
constexpr int kAdjInitThreads = 256;

// words w[0..7] = the 8 floats of vectors (q+sv, q+sv+1); elements R..R+3
template <int R>
__device__ __forceinline__ float4 cut4(const float (&w)[8]) {
    return make_float4(w[R], w[R + 1], w[R + 2], w[R + 3]);
}
__device__ __forceinline__ float4 cut4(const float (&w)[8], int r) {
    switch (r) {
        case 1: return cut4<1>(w);
        case 2: return cut4<2>(w);
        default: return cut4<3>(w);
    }
}

// One adjoint merge level: input row i of level l-1 (grid.x) gathers from the
// level-l gradient rows that read it.  VIN: the gradient rows are 16-byte
// aligned with a pitch multiple of 4 (workspace planes, or the caller's plane
// when ncols % 4 == 0): each read moves as the aligned float4 q + sv of this
// thread plus the next one from the neighbouring lane (warp shuffle; lane 31
// loads its own); else as scalars.  The output is a workspace plane (128-byte
// pitch): float4 stores.
// grid: (rows of level l-1, ceil(ceil(ncols / 4) / (256 * kAdjVecs)))
template <bool VIN>
__global__ void __launch_bounds__(kAdjThreads)
k_fdmt_adj_level(const float* __restrict__ gout, float* __restrict__ gin, const int* __restrict__ off,
                 const int2* __restrict__ ent, int ncols, int out_pitch, int in_pitch) {
    const int i = blockIdx.x;
    const int beg = __ldg(off + i), end = __ldg(off + i + 1);
    const int nv = (ncols + 3) >> 2;
    const int lane = threadIdx.x & 31;
    const int base = blockIdx.y * (kAdjThreads * kAdjVecs) + threadIdx.x;
    float acc[kAdjVecs][4];
#pragma unroll
    for (int k = 0; k < kAdjVecs; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[k][j] = 0.0f;
    for (int e = beg; e < end; ++e) {  // uniform over the block
        const int2 en = __ldg(ent + e);
        const int s = en.y;
        const float* row = gout + static_cast<size_t>(en.x) * out_pitch;
#pragma unroll
        for (int k = 0; k < kAdjVecs; ++k) {
            const int q = base + k * kAdjThreads;
            const int t = 4 * q;
            float v[4];
            if constexpr (VIN) {
                const int sv = s >> 2, r = s & 3;
                const float4* rv = reinterpret_cast<const float4*>(row);
                const int qa = q + sv;
                float4 lo = (qa < nv) ? __ldg(rv + qa) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (r != 0) {
                    float4 hi;
                    hi.x = __shfl_down_sync(0xffffffffu, lo.x, 1);
                    hi.y = __shfl_down_sync(0xffffffffu, lo.y, 1);
                    hi.z = __shfl_down_sync(0xffffffffu, lo.z, 1);
                    hi.w = __shfl_down_sync(0xffffffffu, lo.w, 1);
                    if (lane == 31) hi = (qa + 1 < nv) ? __ldg(rv + qa + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                    lo = cut4(w, r);
                }
                v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = (t + j + s < ncols) ? __ldg(row + t + j + s) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (t + j + s < ncols) acc[k][j] = __fadd_rn(acc[k][j], v[j]);
        }
    }
    float* o = gin + static_cast<size_t>(i) * in_pitch;
#pragma unroll
    for (int k = 0; k < kAdjVecs; ++k) {
        const int q = base + k * kAdjThreads;
        if (q < nv) reinterpret_cast<float4*>(o)[q] = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
    }
}

// Adjoint of level 0 (running means), one window sum and one product per
// level-0 row:
//   gx[c][u] = sum_{r'} RN(1/(r'+1)) * sum_{r=0..r'} [u+r >= r'][u+r < ncols] g0[c,r'][u+r]
// (inner sums r ascending, outer r' ascending).  Thread q owns samples
// 4q..4q+3: each row r' is read as the aligned float4 q plus the next one
// from the lane above (warp shuffle; lane 31 loads its own), which covers
// u + r <= 4q + 7 for up to 5 rows per channel (R0C <= 5; R0C = 0: any
// count, scalar reads).  grid: (ceil(ceil(ncols / 4) / 256), nchan)
template <int R0C>
__global__ void __launch_bounds__(kAdjInitThreads)
k_fdmt_adj_init(const float* __restrict__ g0, float* __restrict__ gx, int ncols, int in_pitch,
                int rows_per_chan, int vec_out) {
    const int c = blockIdx.y;
    const float* g = g0 + static_cast<size_t>(c) * rows_per_chan * in_pitch;
    float* o = gx + static_cast<size_t>(c) * ncols;
    const int nv = (ncols + 3) >> 2;
    const int q = blockIdx.x * kAdjInitThreads + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int u = 4 * q;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const int R = R0C > 0 ? R0C : rows_per_chan;
    for (int rr = 0; rr < R; ++rr) {
        const float* row = g + static_cast<size_t>(rr) * in_pitch;
        const float rcp = __frcp_rn(static_cast<float>(rr + 1));
        float e[8];
        if constexpr (R0C > 0) {
            const float4 lo = (q < nv) ? __ldg(reinterpret_cast<const float4*>(row) + q)
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
            float4 hi;
            hi.x = __shfl_down_sync(0xffffffffu, lo.x, 1);
            hi.y = __shfl_down_sync(0xffffffffu, lo.y, 1);
            hi.z = __shfl_down_sync(0xffffffffu, lo.z, 1);
            hi.w = __shfl_down_sync(0xffffffffu, lo.w, 1);
            if (lane == 31)
                hi = (q + 1 < nv) ? __ldg(reinterpret_cast<const float4*>(row) + q + 1)
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
            e[0] = lo.x; e[1] = lo.y; e[2] = lo.z; e[3] = lo.w;
            e[4] = hi.x; e[5] = hi.y; e[6] = hi.z; e[7] = hi.w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float w = 0.0f;
            const int rmax = R0C > 0 ? R0C : rows_per_chan;
#pragma unroll
            for (int r = 0; r < rmax; ++r) {
                if (r > rr) break;
                const int t = u + j + r;
                if (t >= rr && t < ncols) {
                    float v;
                    if constexpr (R0C > 0) v = e[j + r];
                    else v = __ldg(row + t);
                    w = __fadd_rn(w, v);
                }
            }
            acc[j] = __fadd_rn(acc[j], __fmul_rn(w, rcp));
        }
    }
    if (q >= nv) return;
    if (vec_out && u + 3 < ncols) {
        reinterpret_cast<float4*>(o)[q] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (u + j < ncols) o[u + j] = acc[j];
    }
}

// The last adjoint merge level (level 1 -> level 0) fused with the adjoint of
// level 0 (Keith plans, R0C level-0 rows per channel): for each of channel
// c's level-0 rows the CTA gathers the row's gradient over its samples into
// shared memory (the k_fdmt_adj_level gather of one float4 per thread) and
// folds it into gx at once (the k_fdmt_adj_init sum), so the level-0
// gradient plane is never written or read back.  The sums and their order
// are those of the two kernels, so the bits are too.  CTA b gathers quads
// 255 b .. 255 b + 255 and writes gx for the first 255 of them (each quad's
// window reaches into the next one).  gout: 16-byte aligned rows, pitch a
// multiple of 4.  grid: (ceil(ceil(ncols / 4) / 255), nchan)
template <int R0C>
__global__ void __launch_bounds__(kAdjInitThreads)
k_fdmt_adj_level0(const float* __restrict__ gout, float* __restrict__ gx, const int* __restrict__ off,
                  const int2* __restrict__ ent, int ncols, int out_pitch, int vec_out) {
    constexpr int kOut = kAdjInitThreads - 1;   // quads written per CTA
    __shared__ float4 tile[kAdjInitThreads];
    const int c = blockIdx.y;
    const int nv = (ncols + 3) >> 2;
    const int lane = threadIdx.x & 31;
    const int q = blockIdx.x * kOut + threadIdx.x;
    const int u = 4 * q;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
    for (int rr = 0; rr < R0C; ++rr) {
        const int i = c * R0C + rr;   // level-0 row (c, rr)
        const int beg = __ldg(off + i), end = __ldg(off + i + 1);
        float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int e = beg; e < end; ++e) {  // uniform over the block
            const int2 en = __ldg(ent + e);
            const int s = en.y;
            const float4* rv = reinterpret_cast<const float4*>(gout + static_cast<size_t>(en.x) * out_pitch);
            const int sv = s >> 2, r = s & 3;
            const int qa = q + sv;
            float4 lo = (qa < nv) ? __ldg(rv + qa) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (r != 0) {
                float4 hi;
                hi.x = __shfl_down_sync(0xffffffffu, lo.x, 1);
                hi.y = __shfl_down_sync(0xffffffffu, lo.y, 1);
                hi.z = __shfl_down_sync(0xffffffffu, lo.z, 1);
                hi.w = __shfl_down_sync(0xffffffffu, lo.w, 1);
                if (lane == 31) hi = (qa + 1 < nv) ? __ldg(rv + qa + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                lo = cut4(w, r);
            }
            const float v[4] = {lo.x, lo.y, lo.z, lo.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (u + j + s < ncols) g[j] = __fadd_rn(g[j], v[j]);
        }
        tile[threadIdx.x] = make_float4(g[0], g[1], g[2], g[3]);
        __syncthreads();
        if (threadIdx.x < kOut) {
            const float4 a = tile[threadIdx.x], b = tile[threadIdx.x + 1];
            const float e8[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            const float rcp = __frcp_rn(static_cast<float>(rr + 1));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float w = 0.0f;
#pragma unroll
                for (int r = 0; r < R0C; ++r) {
                    if (r > rr) break;
                    const int t = u + j + r;
                    if (t >= rr && t < ncols) w = __fadd_rn(w, e8[j + r]);
                }
                acc[j] = __fadd_rn(acc[j], __fmul_rn(w, rcp));
            }
        }
        __syncthreads();   // the tile is rewritten for the next row
    }
    if (threadIdx.x >= kOut || q >= nv) return;
    float* o = gx + static_cast<size_t>(c) * ncols;
    if (vec_out && u + 3 < ncols) {
        reinterpret_cast<float4*>(o)[q] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (u + j < ncols) o[u + j] = acc[j];
    }
}

// ---- adjoint run segments (layout and blob: AdjRun, internal.h) ---------------
constexpr int kAdjRunThreads = 256;
constexpr int kAdjRunWarps = kAdjRunThreads / 32;

struct AdjRunArgs {
    const float* in;      // gradient of level l1
    float* out;           // of level l0, or of the channels (FINAL)
    const AdjTile* tiles;
    const int2* rows;
    const int* blob;
    int ncols, in_pitch, out_pitch, nrt, total;
    int pitch_x, y0, blob0, max_blob;
    int vec;              // the input rows' windows start on 16-byte boundaries
};

// A row's sum over K chunks; `at` = the index of its terms in B (a multiple of
// 4) | its kind.  Most rows are two inner sums of two terms, or of one, whose
// loads are all issued before the first add; the others take their terms one
// by one.  (x + 0 turns -0 into the +0 that the sums start from.)
template <int K>
__device__ __forceinline__ void sum_terms(float (&acc)[K], const int* B, int at, const char* lane_base) {
    const int4* q4 = reinterpret_cast<const int4*>(B + (at & ~3));
    const int4 f = *q4;
    const int kind = at & 3;
    if (kind == kAdjPairs || kind == kAdjOnes) {
        float v[4][K];
        load_row<K>(v[0], lane_base + (f.x & 0xffffc));
        load_row<K>(v[1], lane_base + (f.y & 0xffffc));
        if (kind == kAdjPairs) {
            load_row<K>(v[2], lane_base + (f.z & 0xffffc));
            load_row<K>(v[3], lane_base + (f.w & 0xffffc));
            add_rows<K>(v[0], v[0], v[1]);
            add_rows<K>(v[1], v[2], v[3]);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) v[0][k] = __fadd_rn(v[0][k], 0.0f);
        add_rows<K>(acc, v[0], v[1]);
        return;
    }
    float part[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = part[k] = 0.0f;
    if (kind == kAdjZero) return;
    const int* t = B + (at & ~3);
    int q = f.x;
#pragma unroll 1
    for (bool more = true; more;) {
        const int cur = q;
        q = *++t;
        more = (cur & kAdjEnd) == 0;
        float v[K];
        load_row<K>(v, lane_base + (cur & 0xffffc));
        add_rows<K>(part, part, v);
        if (cur & 1) {
            add_rows<K>(acc, acc, part);
#pragma unroll
            for (int k = 0; k < K; ++k) part[k] = 0.0f;
        }
    }
}

// A channel's gradient: per level-0 row r' the sum w of its value g at
// offsets 0..r' (only samples u + r >= r' where the window reaches them),
// times RN(1 / (r' + 1)), rows in ascending order.  u0 = this lane's first
// sample.
template <int K>
__device__ __forceinline__ void sum_channel(float (&gx)[K], const int* B, int at, const char* lane_base, int u0,
                                            bool edge) {
    float part[K], g[K], w[K];
#pragma unroll
    for (int k = 0; k < K; ++k) gx[k] = part[k] = g[k] = w[k] = 0.0f;
    if ((at & 3) == kAdjZero) return;
    const int* t = B + (at & ~3);
    int q = *t;
#pragma unroll 1
    for (bool more = true; more;) {
        const int cur = q;
        q = *++t;
        more = (cur & kAdjEnd) == 0;
        float v[K];
        load_row<K>(v, lane_base + (cur & 0xffffc));
        add_rows<K>(part, part, v);
        if (cur & 1) {
            add_rows<K>(g, g, part);
#pragma unroll
            for (int k = 0; k < K; ++k) part[k] = 0.0f;
        }
        if (cur & 2) {
            const int rr = (cur >> 20) & 7, r = (cur >> 23) & 7;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (!edge || u0 + 32 * k + r >= rr) w[k] = __fadd_rn(w[k], g[k]);
                g[k] = 0.0f;
            }
            if (cur & (1 << 26)) {
                const float rcp = __frcp_rn(static_cast<float>(rr + 1));
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    gx[k] = __fadd_rn(gx[k], __fmul_rn(w[k], rcp));
                    w[k] = 0.0f;
                }
            }
        }
    }
}

// Persistent, two CTAs per SM, tiles and copies as in k_fdmt_run (the next
// tile's input is copied into X while stage 2 reads Y); a warp forms whole
// rows, its share of a stage's rows one after another.
// What bounds it: shared-memory wavefronts, about four loads per row and pair
// of levels and one store, and the loop over the rows that are not two pairs.
// It replaces one gather pass over HBM per level: 1024 x 65536 0.568 ms
// against 1.29 ms, 256 x 24485 60 us against 123 (its odd rows were read one
// sample at a time).  Terms taken one by one for every row: 0.591; two terms
// per turn of the loop: 0.642.
template <bool FINAL>
__global__ void __launch_bounds__(kAdjRunThreads, 2) k_adj_run(const AdjRunArgs a) {
    constexpr int K1 = kRunMidChunks, K2 = kRunOutChunks;
    extern __shared__ __align__(16) float sm[];
    const unsigned sbase = static_cast<unsigned>(__cvta_generic_to_shared(sm));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const char* lane_base = reinterpret_cast<const char*>(sm) + 4 * lane;
    auto tile_of = [&](int rt) {
        const int4* p = reinterpret_cast<const int4*>(a.tiles + rt);
        const int4 lo = __ldg(p), hi = __ldg(p + 1);
        AdjTile t{};
        t.row = lo.x; t.blob = lo.y; t.len = lo.z; t.n_in = lo.w; t.n1 = hi.x; t.n2 = hi.y; t.max_e = hi.z;
        return t;
    };
    auto row_entries = [&](const AdjTile& t) {
        const int j = warp + kAdjRunWarps * lane;
        return j < t.n_in ? __ldg(a.rows + t.row + j) : make_int2(0, 0);
    };
    auto issue = [&](const AdjTile& t, int2 mine, int tt, int eb) {
        const unsigned sb = sbase + 4u * (a.blob0 + eb * a.max_blob);
        for (int i = threadIdx.x; i < (t.len >> 2); i += kAdjRunThreads) copy16(sb + 16u * i, a.blob + t.blob + 4 * i);
        const int t0 = tt * kSegTile;
        if (t0 >= a.ncols + t.max_e) return;   // every output of the tile is past the row's end
        const int pieces = a.pitch_x >> 2;
        for (int i = 0, j = warp; j < t.n_in; ++i, j += kAdjRunWarps) {
            const int row = __shfl_sync(0xffffffffu, mine.x, i), lead = __shfl_sync(0xffffffffu, mine.y, i);
            const int ts = t0 - lead;
            const float* src = a.in + static_cast<size_t>(row) * a.in_pitch + ts;
            float* d = sm + j * a.pitch_x;
            const unsigned dst = sbase + 4u * (j * a.pitch_x);
            if (ts >= a.ncols) {   // wholly past the end
                for (int c = lane; c < pieces; c += 32) reinterpret_cast<float4*>(d)[c] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else if (a.vec && ts >= 0 && ts + a.pitch_x <= a.ncols) {
                const float* s0 = src + 4 * lane;
                const unsigned d0 = dst + 16u * lane;
                copy16(d0, s0);
                copy16(d0 + 512u, s0 + 128);
                if (lane + 64 < pieces) copy16(d0 + 1024u, s0 + 256);
            } else {
                for (int c = lane; c < a.pitch_x; c += 32) {
                    if (ts + c >= 0 && ts + c < a.ncols) copy4(dst + 4u * c, src + c);
                    else d[c] = 0.0f;
                }
            }
        }
    };
    const int G = static_cast<int>(gridDim.x);
    const int gq = G / a.nrt, gr = G % a.nrt;
    int w = blockIdx.x;
    int rt = w % a.nrt, tt = w / a.nrt;
    AdjTile t = tile_of(rt);
    issue(t, row_entries(t), tt, 0);
    for (int eb = 0; w < a.total; eb ^= 1, w += G) {
        const bool more = w + G < a.total;
        int rn = rt + gr, tn = tt + gq;
        if (rn >= a.nrt) { rn -= a.nrt; ++tn; }
        if (!more) rn = rt;
        const AdjTile next = tile_of(rn);
        const int2 next_rows = row_entries(next);
        copy_wait();
        __syncthreads();   // X and the blob are in, every warp is done with Y
        const int t0 = tt * kSegTile;
        const bool live = t0 < a.ncols + t.max_e;
        const int* B = reinterpret_cast<const int*>(sm) + a.blob0 + eb * a.max_blob;
        if (live) {
            const int r0 = t.n1 * warp / kAdjRunWarps, r1 = t.n1 * (warp + 1) / kAdjRunWarps;
            char* dst = reinterpret_cast<char*>(sm + a.y0 + r0 * kRunMid) + 4 * lane;
#pragma unroll 1
            for (int r = r0; r < r1; ++r, dst += 4 * kRunMid) {
                float o[K1];
                sum_terms<K1>(o, B, B[r], lane_base);
#pragma unroll
                for (int k = 0; k < K1; ++k) *reinterpret_cast<float*>(dst + 128 * k) = o[k];
            }
        }
        __syncthreads();   // Y is in, every warp is done with X
        if (more) issue(next, next_rows, tn, eb ^ 1);
        if (live) {
            const int* H = B + t.n1;
            const int r0 = t.n2 * warp / kAdjRunWarps, r1 = t.n2 * (warp + 1) / kAdjRunWarps;
#pragma unroll 1
            for (int r = r0; r < r1; ++r) {
                const int row = H[3 * r], first = t0 - H[3 * r + 1];   // the window's first sample
                if (first >= a.ncols || first + kSegTile <= 0) continue;
                const int u0 = first + lane;
                float o[K2];
                if constexpr (FINAL) sum_channel<K2>(o, B, H[3 * r + 2], lane_base, u0, first < 8);
                else sum_terms<K2>(o, B, H[3 * r + 2], lane_base);
                float* dst = a.out + static_cast<size_t>(row) * a.out_pitch + u0;
                if (first >= 0 && first + kSegTile <= a.ncols) {
#pragma unroll
                    for (int k = 0; k < K2; ++k) dst[32 * k] = o[k];
                } else {
#pragma unroll
                    for (int k = 0; k < K2; ++k)
                        if (u0 + 32 * k >= 0 && u0 + 32 * k < a.ncols) dst[32 * k] = o[k];
                }
            }
        }
        t = next;
        rt = rn;
        tt = tn;
    }
}

template <bool FINAL>
bfs_status launch_adj_run(const AdjRun& ar, const AdjRunArgs& args, cudaStream_t s) {
    auto kern = k_adj_run<FINAL>;
    // opt-in and resident CTAs as for the forward's run segments
    static std::mutex mu;
    static std::map<int, size_t> optin;
    static std::map<std::pair<int, size_t>, int> resident;
    int dev = 0;
    BFS_CUDA(cudaGetDevice(&dev));
    int ctas = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        size_t& have = optin[dev];
        if (have < ar.smem_bytes) {
            BFS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(ar.smem_bytes)));
            have = ar.smem_bytes;
        }
        auto it = resident.find({dev, ar.smem_bytes});
        if (it == resident.end()) {
            int per_sm = 0, sms = 0;
            BFS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kAdjRunThreads, ar.smem_bytes));
            BFS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            if (per_sm < 1) return fail(BFS_ERR_CUDA, "k_adj_run does not fit an SM");
            it = resident.emplace(std::make_pair(dev, ar.smem_bytes), per_sm * sms).first;
        }
        ctas = it->second;
    }
    kern<<<std::min(args.total, ctas), kAdjRunThreads, ar.smem_bytes, s>>>(args);
    BFS_LAUNCH_CHECK("k_adj_run");
    return BFS_OK;
}

// Adjoint of a Pravir plan's level 0 (rows with delays dt_k per channel,
// lvl0 = row cumsum then delays): the same window-mean transpose,
//   gx[c][u] = sum_k RN(1/(dt_k+1)) * sum_{j=0..dt_k} [u+j >= dt_k][u+j < ncols] g0[k][u+j].
// grid: (ceil(ncols / 256), nchan)
__global__ void __launch_bounds__(kAdjInitThreads)
k_fdmt_adj_init_grid(const float* __restrict__ g0, float* __restrict__ gx, const int* __restrict__ lvl0,
                     int nchan, int ncols, int in_pitch) {
    const int c = blockIdx.y;
    const int u = blockIdx.x * kAdjInitThreads + threadIdx.x;
    if (u >= ncols) return;
    const int r0 = __ldg(lvl0 + c), nr = __ldg(lvl0 + c + 1) - r0;
    const int* dts = lvl0 + nchan + 1 + r0;
    float acc = 0.0f;
    for (int k = 0; k < nr; ++k) {
        const int d = __ldg(dts + k);
        const float* row = g0 + static_cast<size_t>(r0 + k) * in_pitch;
        float w = 0.0f;
        for (int j = 0; j <= d; ++j) {
            const int t = u + j;
            if (t >= d && t < ncols) w = __fadd_rn(w, __ldg(row + t));
        }
        acc = __fadd_rn(acc, __fmul_rn(w, __frcp_rn(static_cast<float>(d + 1))));
    }
    gx[static_cast<size_t>(c) * ncols + u] = acc;
}

// S/N at cells: cells[3k..3k+2] = {row, start, width}.  A cell outside the
// plane gives NaN.
__global__ void k_snr_cells(const float* __restrict__ plane, int rows, int cols,
                            const float* __restrict__ stats, const int* __restrict__ cells, int n,
                            float* __restrict__ snr) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int d = cells[3 * k], t = cells[3 * k + 1], w = cells[3 * k + 2];
    if (d < 0 || d >= rows || t < 0 || w < 1 || w > cols - t) { snr[k] = __int_as_float(0x7fc00000); return; }
    const float m = stats[d], sd = stats[rows + d];
    const float* x = plane + static_cast<size_t>(d) * cols + t;
    float sum = 0.0f;
    for (int j = 0; j < w; ++j)
        sum = __fadd_rn(sum, sd > 0.0f ? __fdiv_rn(__fsub_rn(__ldg(x + j), m), sd) : 0.0f);
    snr[k] = __fdiv_rn(sum, __fsqrt_rn(static_cast<float>(w)));
}

// Gradient of sum_k gsnr[k] * S_k with respect to the plane: each CTA writes
// one of gridDim.y parts of a row; its warp 0 collects the row's cells in
// cell order (ballot compaction, up to kMaxCellsPerRow) and the row constants;
// then every sample of the part is written (rows without cells get zeros).
// HBM-bound by the stores; a row with cells is a chain of loads and stores,
// so it is cut into parts and each thread keeps four 16-byte groups (VEC:
// rows 16-byte aligned) or four samples in flight.  1024 x 65536, 8 cells:
// 184 us with one CTA per row and one sample at a time.
constexpr int kMaxCellsPerRow = 512;
constexpr int kSnrThreads = 256;
constexpr int kSnrPart = 8192;   // samples per CTA

template <bool VEC>
__global__ void __launch_bounds__(kSnrThreads)
k_snr_cells_adjoint(const float* __restrict__ plane, int rows, int cols, const float* __restrict__ stats,
                    const int* __restrict__ cells, int n, const float* __restrict__ snr,
                    const float* __restrict__ gsnr, float* __restrict__ gplane, int* __restrict__ err) {
    __shared__ int s_t[kMaxCellsPerRow], s_w[kMaxCellsPerRow];
    __shared__ float s_c[kMaxCellsPerRow];  // gsnr / (sd sqrt(w))
    __shared__ int s_n;
    __shared__ float s_a, s_b;              // constant term, coefficient of (y - m)
    const int d = blockIdx.x;
    const float m = stats[d], sd = stats[rows + d];
    const float nf = static_cast<float>(cols);
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int cnt = 0;
        float a = 0.0f, b = 0.0f;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + lane;
            const bool mine = k < n && cells[3 * k] == d;
            const unsigned bal = __ballot_sync(0xffffffffu, mine);
            if (mine) {
                const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
                if (pos < kMaxCellsPerRow) {
                    const int w = cells[3 * k + 2];
                    s_t[pos] = cells[3 * k + 1];
                    s_w[pos] = w;
                    s_c[pos] = sd > 0.0f ? gsnr[k] / (sd * sqrtf(static_cast<float>(w))) : 0.0f;
                }
            }
            cnt += __popc(bal);
        }
        __syncwarp();
        if (lane == 0) {
            if (cnt > kMaxCellsPerRow) atomicExch(err, 1);
            cnt = min(cnt, kMaxCellsPerRow);
            // row constants in cell order: sum_k -w_k c_k / N and -gsnr_k S_k / (N sd^2)
            int j = 0;
            for (int k = 0; k < n && j < cnt; ++k) {
                if (cells[3 * k] != d) continue;
                a += -static_cast<float>(s_w[j]) * s_c[j] / nf;
                if (sd > 0.0f) b += -gsnr[k] * snr[k] / (nf * sd * sd);
                ++j;
            }
            s_n = cnt;
            s_a = a;
            s_b = b;
        }
    }
    __syncthreads();
    const int cnt = s_n;
    const float a = s_a, b = s_b;
    const float* y = plane + static_cast<size_t>(d) * cols;
    float* g = gplane + static_cast<size_t>(d) * cols;
    const int beg = blockIdx.y * kSnrPart, end = min(cols, beg + kSnrPart);
    auto value = [&](int u, float yu) {
        float v = a + b * (yu - m);
        for (int j = 0; j < cnt; ++j)
            if (u >= s_t[j] && u < s_t[j] + s_w[j]) v += s_c[j];
        return v;
    };
    constexpr int kStep = VEC ? 4 : 1, kFly = 4;
    for (int u0 = beg + kStep * threadIdx.x; u0 < end; u0 += kStep * kFly * kSnrThreads) {
        if constexpr (VEC) {   // (cols a multiple of 4: a group lies wholly inside or outside the row)
            float4 q[kFly];
#pragma unroll
            for (int k = 0; k < kFly; ++k) {
                const int u = u0 + 4 * k * kSnrThreads;
                q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (cnt > 0 && u < end) q[k] = __ldg(reinterpret_cast<const float4*>(y + u));
            }
#pragma unroll
            for (int k = 0; k < kFly; ++k) {
                const int u = u0 + 4 * k * kSnrThreads;
                if (u >= end) break;
                if (cnt > 0)
                    q[k] = make_float4(value(u, q[k].x), value(u + 1, q[k].y), value(u + 2, q[k].z), value(u + 3, q[k].w));
                *reinterpret_cast<float4*>(g + u) = q[k];
            }
        } else {
            float q[kFly];
#pragma unroll
            for (int k = 0; k < kFly; ++k) {
                const int u = u0 + k * kSnrThreads;
                q[k] = cnt > 0 && u < end ? __ldg(y + u) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < kFly; ++k) {
                const int u = u0 + k * kSnrThreads;
                if (u < end) g[u] = cnt > 0 ? value(u, q[k]) : 0.0f;
            }
        }
    }
}

inline int plane_pitch4(int ncols) { return (ncols + 31) / 32 * 32; }

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

// Rows of the adjoint's ping-pong planes: level l-1's gradient (l = niter..1)
// lives in buffer (l-1) & 1; the level-niter gradient is the caller's plane.
void adjoint_plane_rows(const FdmtPlanHost& h, size_t rows[2]) {
    rows[0] = rows[1] = 0;
    for (int l = 0; l < h.niter; ++l)
        rows[l & 1] = std::max(rows[l & 1], static_cast<size_t>(h.lv[l].total_rows()));
}

size_t adjoint_ws_bytes(const FdmtPlanHost& h) {
    size_t rows[2];
    adjoint_plane_rows(h, rows);
    const size_t P = plane_pitch4(h.ncols);
    return align256(rows[0] * P * sizeof(float)) + align256(rows[1] * P * sizeof(float));
}

constexpr size_t kAdjRunSmem = 113 * 1024;   // two CTAs per SM

// The plan's levels as adjoint run segments of two to four levels, from the
// top down; empty where one does not fit (one gather pass per level then).
// Outputs per tile: as many as fit; fewer where all tiles would run at once.
void plan_adjoint_runs(const FdmtPlanHost& h, const AdjointTables& tab, std::vector<AdjRun>* out) {
    out->clear();
    if (h.niter < 2) return;
    const int nseg = (h.niter + 3) / 4;
    size_t rows[2];
    adjoint_plane_rows(h, rows);
    int l1 = h.niter;
    for (int i = 0; i < nseg; ++i) {
        const int l0 = l1 - (h.niter / nseg + (i < h.niter % nseg ? 1 : 0));
        const bool final = l0 == 0 && h.kind == BFS_PLAN_KEITH && h.rows_per_chan0 <= 5;
        if (!final && static_cast<size_t>(h.lv[l0].total_rows()) > rows[(nseg - 1 - i) & 1]) {
            out->clear();
            return;
        }
        const int in_pitch = l1 == h.niter ? h.ncols : plane_pitch4(h.ncols);
        const long long tt = (h.ncols + kSegTile - 1) / kSegTile;
        const int outputs = final ? h.nchan : h.lv[l0].total_rows();
        std::vector<int> per_tile;
        for (int G = 48; G >= 8; G -= 4)
            if (G <= 12 || outputs / G * tt >= 2 * 148) per_tile.push_back(G);
        AdjRun ar;
        if (!build_adj_run(h, tab, l0, l1, final, per_tile, in_pitch, kAdjRunSmem, &ar)) {
            out->clear();
            return;
        }
        out->push_back(std::move(ar));
        l1 = l0;
    }
}

bfs_status ensure_adjoint_tables(bfs_fdmt_plan* p) {
    if (p->d_adj_tables) return BFS_OK;
    if (!p->adj.built) {
        build_adjoint_tables(p->host, &p->adj);
        plan_adjoint_runs(p->host, p->adj, &p->adj_runs);
    }
    const AdjointTables& A = p->adj;
    TableUpload up;
    std::vector<int2> pairs;
    std::vector<AdjTile> tiles;
    std::vector<int> rows, blob;
    p->adj_run0.clear();
    for (const AdjRun& r : p->adj_runs) {
        p->adj_run0.push_back({tiles.size(), rows.size(), blob.size()});
        tiles.insert(tiles.end(), r.tiles.begin(), r.tiles.end());
        rows.insert(rows.end(), r.rows.begin(), r.rows.end());
        blob.insert(blob.end(), r.blob.begin(), r.blob.end());
    }
    up.add(&p->d_adj_tiles, tiles);
    up.add(&p->d_adj_rows, rows);
    up.add(&p->d_adj_blob, blob);
    if (p->adj_runs.empty()) {   // one gather pass per level
        for (size_t i = 0; i + 1 < A.ent.size(); i += 2) pairs.push_back(make_int2(A.ent[i], A.ent[i + 1]));
        up.add(&p->d_adj_off, A.off);
        up.add(&p->d_adj_ent, pairs);
    }
    return up.commit(&p->d_adj_tables);
}

bfs_status adjoint_run(bfs_fdmt_plan* p, const float* d_gy, float* d_gx, float* buf0, float* buf1,
                       cudaStream_t s) {
    const FdmtPlanHost& h = p->host;
    const int T = h.ncols;
    const int P = plane_pitch4(T);
    float* bufs[2] = {buf0, buf1};
    const size_t nrun = p->adj_runs.size();
    for (size_t i = 0; i < nrun; ++i) {
        const AdjRun& ar = p->adj_runs[i];
        AdjRunArgs a;
        a.in = i == 0 ? d_gy : bufs[(nrun - i) & 1];
        a.out = ar.final ? d_gx : bufs[(nrun - 1 - i) & 1];
        a.tiles = p->d_adj_tiles + p->adj_run0[i][0];
        a.rows = reinterpret_cast<const int2*>(p->d_adj_rows + p->adj_run0[i][1]);
        a.blob = p->d_adj_blob + p->adj_run0[i][2];
        a.ncols = T;
        a.in_pitch = i == 0 ? T : P;
        a.out_pitch = ar.final ? T : P;
        a.nrt = static_cast<int>(ar.tiles.size());
        const long long total = static_cast<long long>(a.nrt) * ((T + ar.max_e + kSegTile - 1) / kSegTile);
        BFS_ARG(total <= (1LL << 30), "too many adjoint tiles");
        a.total = static_cast<int>(total);
        a.pitch_x = ar.pitch_x; a.y0 = ar.y0; a.blob0 = ar.blob0; a.max_blob = ar.max_blob;
        a.vec = (reinterpret_cast<uintptr_t>(a.in) & 15) == 0 ? 1 : 0;
        bfs_status st = ar.final ? launch_adj_run<true>(ar, a, s) : launch_adj_run<false>(ar, a, s);
        if (st != BFS_OK) return st;
    }
    if (nrun > 0 && p->adj_runs.back().final) return BFS_OK;
    const int span = kAdjThreads * kAdjVecs;
    const int gy_blocks = ((T + 3) / 4 + span - 1) / span;
    BFS_ARG(gy_blocks <= 65535, "ncols too large for this build");
    // Keith plans: the last merge level runs fused with the level-0 adjoint
    // when the level-1 gradient rows allow 16-byte reads
    const int r0c = h.rows_per_chan0;
    const float* src1 = (h.niter == 1) ? d_gy : bufs[1];
    const int pitch1 = (h.niter == 1) ? T : P;
    const bool fuse0 = nrun == 0 && h.kind == BFS_PLAN_KEITH && r0c >= 1 && r0c <= 5 && pitch1 % 4 == 0 &&
                       (reinterpret_cast<uintptr_t>(src1) & 15) == 0 &&
                       h.lv[0].total_rows() == h.nchan * r0c;
    for (int l = nrun > 0 ? 0 : h.niter; l >= (fuse0 ? 2 : 1); --l) {
        const float* src = (l == h.niter) ? d_gy : bufs[l & 1];
        float* dst = bufs[(l - 1) & 1];
        const int in_pitch = (l == h.niter) ? T : P;
        const int rows_in = h.lv[l - 1].total_rows();
        const int* off = p->d_adj_off + p->adj.off_pos[l];
        const int2* ent = p->d_adj_ent + p->adj.ent_pos[l];
        dim3 grid(rows_in, gy_blocks);
        const bool vin = (in_pitch % 4 == 0) && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
        if (vin)
            k_fdmt_adj_level<true><<<grid, kAdjThreads, 0, s>>>(src, dst, off, ent, T, in_pitch, P);
        else
            k_fdmt_adj_level<false><<<grid, kAdjThreads, 0, s>>>(src, dst, off, ent, T, in_pitch, P);
        BFS_LAUNCH_CHECK("k_fdmt_adj_level");
    }
    if (h.kind == BFS_PLAN_PRAVIR) {
        dim3 g2((T + kAdjInitThreads - 1) / kAdjInitThreads, h.nchan);
        BFS_ARG(g2.y <= 65535, "nchan too large for this build");
        k_fdmt_adj_init_grid<<<g2, kAdjInitThreads, 0, s>>>(bufs[0], d_gx, p->d_lvl0, h.nchan, T, P);
        BFS_LAUNCH_CHECK("k_fdmt_adj_init_grid");
        return BFS_OK;
    }
    const int vec_out = (T % 4 == 0) && (reinterpret_cast<uintptr_t>(d_gx) & 15) == 0;
    if (fuse0) {
        const int* off = p->d_adj_off + p->adj.off_pos[1];
        const int2* ent = p->d_adj_ent + p->adj.ent_pos[1];
        dim3 g0(((T + 3) / 4 + kAdjInitThreads - 2) / (kAdjInitThreads - 1), h.nchan);
        BFS_ARG(g0.y <= 65535, "nchan too large for this build");
        switch (r0c) {
            case 1: k_fdmt_adj_level0<1><<<g0, kAdjInitThreads, 0, s>>>(src1, d_gx, off, ent, T, pitch1, vec_out); break;
            case 2: k_fdmt_adj_level0<2><<<g0, kAdjInitThreads, 0, s>>>(src1, d_gx, off, ent, T, pitch1, vec_out); break;
            case 3: k_fdmt_adj_level0<3><<<g0, kAdjInitThreads, 0, s>>>(src1, d_gx, off, ent, T, pitch1, vec_out); break;
            case 4: k_fdmt_adj_level0<4><<<g0, kAdjInitThreads, 0, s>>>(src1, d_gx, off, ent, T, pitch1, vec_out); break;
            default: k_fdmt_adj_level0<5><<<g0, kAdjInitThreads, 0, s>>>(src1, d_gx, off, ent, T, pitch1, vec_out); break;
        }
        BFS_LAUNCH_CHECK("k_fdmt_adj_level0");
        return BFS_OK;
    }
    dim3 grid(((T + 3) / 4 + kAdjInitThreads - 1) / kAdjInitThreads, h.nchan);
    BFS_ARG(grid.y <= 65535, "nchan too large for this build");
    switch (h.rows_per_chan0) {
        case 1: k_fdmt_adj_init<1><<<grid, kAdjInitThreads, 0, s>>>(bufs[0], d_gx, T, P, 1, vec_out); break;
        case 2: k_fdmt_adj_init<2><<<grid, kAdjInitThreads, 0, s>>>(bufs[0], d_gx, T, P, 2, vec_out); break;
        case 3: k_fdmt_adj_init<3><<<grid, kAdjInitThreads, 0, s>>>(bufs[0], d_gx, T, P, 3, vec_out); break;
        case 4: k_fdmt_adj_init<4><<<grid, kAdjInitThreads, 0, s>>>(bufs[0], d_gx, T, P, 4, vec_out); break;
        case 5: k_fdmt_adj_init<5><<<grid, kAdjInitThreads, 0, s>>>(bufs[0], d_gx, T, P, 5, vec_out); break;
        default:
            k_fdmt_adj_init<0><<<grid, kAdjInitThreads, 0, s>>>(bufs[0], d_gx, T, P, h.rows_per_chan0, vec_out);
    }
    BFS_LAUNCH_CHECK("k_fdmt_adj_init");
    return BFS_OK;
}

}  // namespace
}  // namespace bfs

using namespace bfs;

extern "C" bfs_status bfs_fdmt_plan_adjoint_run(const bfs_fdmt_plan* plan, int pass, int* params, int* tiles,
                                                int tiles_cap, int* rows, int rows_cap, int* blob, int blob_cap) {
    BFS_ARG(plan != nullptr && params != nullptr, "null argument");
    AdjointTables tab;
    std::vector<AdjRun> runs;
    build_adjoint_tables(plan->host, &tab);
    plan_adjoint_runs(plan->host, tab, &runs);
    params[0] = static_cast<int>(runs.size());
    if (pass < 0 || pass >= params[0]) return BFS_OK;
    const AdjRun& ar = runs[pass];
    constexpr int ti = static_cast<int>(sizeof(AdjTile) / sizeof(int));
    const int v[12] = {params[0], ar.l0, ar.l1, ar.final ? 1 : 0, ar.pitch_x, ar.y0, ar.blob0, ar.max_blob, ar.max_e,
                       static_cast<int>(ar.tiles.size()), static_cast<int>(ar.rows.size() / 2),
                       static_cast<int>(ar.blob.size())};
    std::copy(v, v + 12, params);
    if (tiles) {
        BFS_ARG(tiles_cap >= ti * v[9], "tiles needs %d ints", ti * v[9]);
        std::memcpy(tiles, ar.tiles.data(), ar.tiles.size() * sizeof(AdjTile));
    }
    if (rows) {
        BFS_ARG(rows_cap >= 2 * v[10], "rows needs %d ints", 2 * v[10]);
        std::copy(ar.rows.begin(), ar.rows.end(), rows);
    }
    if (blob) {
        BFS_ARG(blob_cap >= v[11], "blob needs %d ints", v[11]);
        std::copy(ar.blob.begin(), ar.blob.end(), blob);
    }
    return BFS_OK;
}

extern "C" bfs_status bfs_fdmt_adjoint_workspace_size(const bfs_fdmt_plan* plan, size_t* bytes) {
    BFS_ARG(plan != nullptr && bytes != nullptr, "null argument");
    *bytes = adjoint_ws_bytes(plan->host);
    return BFS_OK;
}

extern "C" bfs_status bfs_fdmt_adjoint_ws(bfs_fdmt_plan* plan, const float* d_grad_out, float* d_grad_in,
                                          void* d_workspace, size_t workspace_bytes, void* stream) {
    BFS_ARG(plan != nullptr && d_grad_out != nullptr && d_grad_in != nullptr, "null argument");
    BFS_ARG(!plan->host_only, "plan was created with bfs_fdmt_plan_create_host");
    const size_t need = adjoint_ws_bytes(plan->host);
    BFS_ARG(d_workspace != nullptr && workspace_bytes >= need,
            "workspace of %zu bytes is smaller than the %zu needed", workspace_bytes, need);
    BFS_ARG((reinterpret_cast<uintptr_t>(d_workspace) & 255) == 0, "workspace must be 256-byte aligned");
    bfs_status st = ensure_adjoint_tables(plan);
    if (st != BFS_OK) return st;
    size_t rows[2];
    adjoint_plane_rows(plan->host, rows);
    char* w = static_cast<char*>(d_workspace);
    float* b0 = reinterpret_cast<float*>(w);
    float* b1 = reinterpret_cast<float*>(w + align256(rows[0] * plane_pitch4(plan->host.ncols) * sizeof(float)));
    return adjoint_run(plan, d_grad_out, d_grad_in, b0, b1, as_stream(stream));
}

extern "C" bfs_status bfs_fdmt_adjoint(bfs_fdmt_plan* plan, const float* d_grad_out, float* d_grad_in,
                                       void* stream) {
    BFS_ARG(plan != nullptr && d_grad_out != nullptr && d_grad_in != nullptr, "null argument");
    BFS_ARG(!plan->host_only, "plan was created with bfs_fdmt_plan_create_host");
    bfs_status st = ensure_adjoint_tables(plan);
    if (st != BFS_OK) return st;
    size_t rows[2];
    adjoint_plane_rows(plan->host, rows);
    if (!plan->adj_runs.empty()) {   // only the planes between the segments reach HBM
        rows[0] = rows[1] = 0;
        const size_t n = plan->adj_runs.size();
        for (size_t i = 0; i < n; ++i)
            if (!plan->adj_runs[i].final)
                rows[(n - 1 - i) & 1] = std::max<size_t>(rows[(n - 1 - i) & 1],
                                                         plan->host.lv[plan->adj_runs[i].l0].total_rows());
    }
    const size_t P = plane_pitch4(plan->host.ncols);
    for (int b = 0; b < 2; ++b) {
        if (plan->d_adj_buf[b] || rows[b] == 0) continue;
        cudaError_t e = cudaMalloc(&plan->d_adj_buf[b], rows[b] * P * sizeof(float));
        if (e != cudaSuccess) {
            cudaGetLastError();
            plan->d_adj_buf[b] = nullptr;
            return fail(BFS_ERR_ALLOC, "cudaMalloc for an adjoint FDMT plane failed: %s", cudaGetErrorString(e));
        }
    }
    return adjoint_run(plan, d_grad_out, d_grad_in, static_cast<float*>(plan->d_adj_buf[0]),
                       static_cast<float*>(plan->d_adj_buf[1]), as_stream(stream));
}

extern "C" bfs_status bfs_boxcar_snr_cells(const float* d_plane, int rows, int cols, const float* d_stats,
                                           const int* d_cells, int n, float* d_snr, void* stream) {
    BFS_ARG(d_plane && d_stats && (n == 0 || (d_cells && d_snr)), "null argument");
    BFS_ARG(rows >= 1 && cols >= 1 && n >= 0, "bad shape");
    if (n == 0) return BFS_OK;
    k_snr_cells<<<(n + 127) / 128, 128, 0, as_stream(stream)>>>(d_plane, rows, cols, d_stats, d_cells, n, d_snr);
    BFS_LAUNCH_CHECK("k_snr_cells");
    return BFS_OK;
}

extern "C" bfs_status bfs_boxcar_snr_cells_adjoint(const float* d_plane, int rows, int cols,
                                                   const float* d_stats, const int* d_cells, int n,
                                                   const float* d_snr, const float* d_gsnr,
                                                   float* d_gplane, void* stream) {
    BFS_ARG(d_plane && d_stats && d_gplane && (n == 0 || (d_cells && d_snr && d_gsnr)), "null argument");
    BFS_ARG(rows >= 1 && cols >= 1 && n >= 0, "bad shape");
    cudaStream_t s = as_stream(stream);
    BFS_ARG((cols + kSnrPart - 1) / kSnrPart <= 65535, "ncols too large for this build");
    const bool vec = cols % 4 == 0 && ((reinterpret_cast<uintptr_t>(d_plane) | reinterpret_cast<uintptr_t>(d_gplane)) & 15) == 0;
    const dim3 grid(rows, (cols + kSnrPart - 1) / kSnrPart);
    auto launch = [&](int* err) {
        if (vec)
            k_snr_cells_adjoint<true><<<grid, kSnrThreads, 0, s>>>(d_plane, rows, cols, d_stats, d_cells, n, d_snr, d_gsnr,
                                                                   d_gplane, err);
        else
            k_snr_cells_adjoint<false><<<grid, kSnrThreads, 0, s>>>(d_plane, rows, cols, d_stats, d_cells, n, d_snr, d_gsnr,
                                                                    d_gplane, err);
        return cudaGetLastError();
    };
    if (n <= kMaxCellsPerRow) {   // no row can hold too many: nothing to read back
        BFS_CUDA(launch(nullptr));
        return BFS_OK;
    }
    int* err = nullptr;
    bfs_status st = stream_alloc(reinterpret_cast<void**>(&err), sizeof(int), s);
    if (st != BFS_OK) return st;
    BFS_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    BFS_CUDA(launch(err));
    int h_err = 0;
    BFS_CUDA(cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    BFS_CUDA(cudaFreeAsync(err, s));
    BFS_CUDA(cudaStreamSynchronize(s));
    BFS_ARG(h_err == 0, "more than %d cells in one row", kMaxCellsPerRow);
    return BFS_OK;
}
