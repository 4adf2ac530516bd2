// Run segments of the FDMT (sm_100a): two to four merge levels per pass over
// HBM, two levels per shared-memory round trip.  The tables and the shared
// layout are described with RunPlan (internal.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "divide.cuh"
#include "fdmt_run.h"
#include "row_ops.cuh"

namespace bfs {
namespace {

constexpr int kRunThreads = 256;
constexpr int kRunWarps = kRunThreads / 32;

// Level-0 row R of a channel (the reference's running mean, one rounding per
// operation) from its samples: p addresses x[t] of this lane's first column.
// POS: -0.0 samples count as +0 (RunPlan::positive).
template <int R, int K, bool POS>
__device__ __forceinline__ void mean_row(float (&v)[K], const char* p) {
    auto samples = [](float (&x)[K], const char* at) {
        load_row<K>(x, at);
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (POS) x[k] = __fadd_rn(x[k], 0.0f);
    };
    samples(v, p);
#pragma unroll
    for (int r = 1; r <= R; ++r) {
        float x[K];
        samples(x, p - 4 * r);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float m = r == 1 ? v[k] : __fmul_rn(v[k], static_cast<float>(r));
            v[k] = div_small(__fadd_rn(m, x[k]), r + 1);
        }
    }
}

struct RunArgs {
    const float* in;
    float* out;
    const RunTile* tiles;
    const int2* rows;
    const int4* ent;
    int ncols, in_pitch, out_pitch, nrt, total;
    int pitch_x, zero_x, zero_y, y0, ent0, max_ent, edge;
    int vec;   // the input rows' windows start on 16-byte boundaries
    int ones;  // the input is all ones (normalisation mode): no loads
};

// An input of stage 1 of an input segment: the level-0 row its entry names; `edge` tiles hold samples before the row number, where the
// level-0 row is 0 (and -0.0 before sample 0, as everywhere).
template <int R0C, int K, bool POS>
__device__ __forceinline__ void load_input(float (&v)[K], const char* lane_base, int q, bool edge, const RunArgs& a,
                                           const RunTile& t, int t0) {
    const int off = q & 0xffffc, r = q >> 20;
    const char* p = lane_base + off;
    switch (r) {
        case 0:   // (the -0.0 row stays as it is)
            if (POS && off != 4 * a.zero_x) mean_row<0, K, true>(v, p);
            else load_row<K>(v, p);
            break;
        case 1: mean_row<1, K, POS>(v, p); break;
        case 2: if constexpr (R0C > 2) mean_row<2, K, POS>(v, p); break;
        case 3: if constexpr (R0C > 3) mean_row<3, K, POS>(v, p); break;
        default: if constexpr (R0C > 4) mean_row<4, K, POS>(v, p); break;
    }
    if (edge && (POS || r > 0) && off != 4 * a.zero_x) {
        const int j = (off >> 2) / a.pitch_x;
        const int first = t0 - __ldg(&a.rows[t.row + j].y) + (off >> 2) - j * a.pitch_x + (threadIdx.x & 31);
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (first + 32 * k < r) v[k] = first + 32 * k < 0 ? -0.0f : 0.0f;
    }
}

// What bounds it: shared-memory wavefronts.  A row formed one level at a time
// costs two loads and a store per 32 columns and level; here a row of two
// levels costs four loads less the ones kept from the row before (2.9 on
// average at 32 rows per tile) and one store, so 1.95 per level against 3.
// 4096 x 45001 in three passes of four levels: 1.04 ms (4.4 TB/s of the 4.6
// GB its schedule moves) against 2.04 ms for the one-level kernel's best
// schedule; 1024 x 65536 0.36 against 0.67, 512 x 32768 0.115 against 0.160.
// With the copies left out a pass of the first shape takes 270 of 369 us,
// with the stages left out 170: the two CTAs of an SM overlap them in part.
// Measured and not kept: more warps (384 or 512 threads: 16 kept columns of
// four inputs do not fit 80 registers; keeping the two sums instead of the
// four inputs 1.07 ms), predicated loads instead of branches (1.13), the next
// tile's rows prefetched into L2 during stage 1 (1.10).
// Persistent: CTA b runs tiles b, b + gridDim.x, ... (tile w = row tile
// w % nrt at time tile w / nrt, so neighbouring CTAs share input rows through
// L2), two CTAs per SM.  A warp forms consecutive rows, lanes on consecutive
// columns: every shared access is one wavefront whatever the offsets.  The
// next tile's input is copied into X while stage 2 reads Y.
template <int S1, int S2, int R0C, bool POS>
__global__ void __launch_bounds__(kRunThreads, 2) k_fdmt_run(const RunArgs a) {
    constexpr int K1 = kRunMidChunks, K2 = kRunOutChunks;
    extern __shared__ __align__(16) float sm[];
    const unsigned sbase = static_cast<unsigned>(__cvta_generic_to_shared(sm));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const char* lane_base = reinterpret_cast<const char*>(sm) + 4 * lane;
    for (int i = threadIdx.x; i < kRunMid; i += kRunThreads) sm[a.zero_x + i] = -0.0f;
    for (int i = threadIdx.x; i < kSegTile; i += kRunThreads) sm[a.zero_y + i] = -0.0f;

    auto tile_of = [&](int rt) {
        const int4* p = reinterpret_cast<const int4*>(a.tiles + rt);
        const int4 lo = __ldg(p), hi = __ldg(p + 1);
        RunTile t{};
        t.row = lo.x; t.ent = lo.y; t.n_in = lo.z; t.n1 = lo.w; t.n2 = hi.x; t.out0 = hi.y;
        return t;
    };
    // this warp's input rows are warp, warp + 8, ..: lane i holds the i-th one's {row, lead}
    auto row_entries = [&](const RunTile& t) {
        const int j = warp + kRunWarps * lane;
        return j < t.n_in ? __ldg(a.rows + t.row + j) : make_int2(0, 0);
    };
    auto issue = [&](const RunTile& t, int2 mine, int tt, int eb) {
        const int nent = t.n1 + t.n2;
        const unsigned se = sbase + 4u * a.ent0 + 16u * eb * a.max_ent;
        for (int i = threadIdx.x; i < nent; i += kRunThreads) copy16(se + 16u * i, a.ent + t.ent + i);
        const int t0 = tt * kSegTile;
        const int pieces = a.pitch_x >> 2;
        for (int i = 0, j = warp; j < t.n_in; ++i, j += kRunWarps) {
            const int row = __shfl_sync(0xffffffffu, mine.x, i), lead = __shfl_sync(0xffffffffu, mine.y, i);
            const int ts = t0 - lead;
            const float* src = a.in + static_cast<size_t>(row) * a.in_pitch + ts;
            float* d = sm + j * a.pitch_x;
            const unsigned dst = sbase + 4u * (j * a.pitch_x);
            if (ts + a.pitch_x <= 0) {   // wholly before sample 0
                const float4 z = make_float4(-0.0f, -0.0f, -0.0f, -0.0f);
                for (int c = lane; c < pieces; c += 32) reinterpret_cast<float4*>(d)[c] = z;
            } else if (a.ones) {
                for (int c = lane; c < a.pitch_x; c += 32) d[c] = ts + c < 0 ? -0.0f : 1.0f;
            } else if (a.vec && ts >= 0 && ts + a.pitch_x <= a.ncols) {
                const float* s0 = src + 4 * lane;
                const unsigned d0 = dst + 16u * lane;
                copy16(d0, s0);
                copy16(d0 + 512u, s0 + 128);
                if (lane + 64 < pieces) copy16(d0 + 1024u, s0 + 256);
            } else {
                for (int c = lane; c < a.pitch_x; c += 32) {
                    if (ts + c < 0) d[c] = -0.0f;
                    else if (ts + c < a.ncols) copy4(dst + 4u * c, src + c);
                    else d[c] = 0.0f;
                }
            }
        }
    };

    const int G = static_cast<int>(gridDim.x);
    const int gq = G / a.nrt, gr = G % a.nrt;   // stepping by gridDim.x without dividing per tile
    int w = blockIdx.x;
    int rt = w % a.nrt, tt = w / a.nrt;
    RunTile t = tile_of(rt);
    issue(t, row_entries(t), tt, 0);
    for (int eb = 0; w < a.total; eb ^= 1, w += G) {
        const bool more = w + G < a.total;
        int rn = rt + gr, tn = tt + gq;
        if (rn >= a.nrt) { rn -= a.nrt; ++tn; }
        if (!more) rn = rt;
        const RunTile next = tile_of(rn);
        const int2 next_rows = row_entries(next);
        copy_wait();
        __syncthreads();   // X and the entries are in, every warp is done with Y
        const int t0 = tt * kSegTile;
        const int4* e = reinterpret_cast<const int4*>(sm + a.ent0) + eb * a.max_ent;
        {
            const bool edge = R0C > 1 && t0 < a.edge;
            const int r0 = t.n1 * warp / kRunWarps, r1 = t.n1 * (warp + 1) / kRunWarps;
            char* dst = reinterpret_cast<char*>(sm + a.y0 + r0 * kRunMid) + 4 * lane;
            float v[2 * S1][K1];
            int4 q4 = e[r0];
            q4 = make_int4(q4.x | 1, q4.y | 1, q4.z | 1, q4.w | 1);   // a warp's first row reads all its inputs
#pragma unroll 1
            for (int r = r0; r < r1; ++r, dst += 4 * kRunMid) {
                const int q[4] = {q4.x, q4.y, q4.z, q4.w};
                q4 = e[r + 1];
#pragma unroll
                for (int i = 0; i < 2 * S1; ++i) {
                    if (q[i] & 1) {
                        if constexpr (R0C <= 1) load_row<K1>(v[i], lane_base + (q[i] - 1));
                        else load_input<R0C, K1, POS>(v[i], lane_base, q[i], edge, a, t, t0);
                    }
                }
                float o[K1];
                add_rows<K1>(o, v[0], v[1]);
                if constexpr (S1 == 2) {
                    float h[K1];
                    add_rows<K1>(h, v[2], v[3]);
                    add_rows<K1>(o, o, h);
                }
#pragma unroll
                for (int k = 0; k < K1; ++k) *reinterpret_cast<float*>(dst + 128 * k) = o[k];
            }
        }
        __syncthreads();   // Y is in, every warp is done with X
        if (more) issue(next, next_rows, tn, eb ^ 1);
        {
            const bool clean = t0 + kSegTile <= a.ncols;
            e += t.n1;
            const int r0 = t.n2 * warp / kRunWarps, r1 = t.n2 * (warp + 1) / kRunWarps;
            float* dst = a.out + static_cast<size_t>(t.out0 + r0) * a.out_pitch + t0 + lane;
            float v[2 * S2][K2];
            int4 q4 = e[r0];
            q4 = make_int4(q4.x | 1, q4.y | 1, q4.z | 1, q4.w | 1);
#pragma unroll 1
            for (int r = r0; r < r1; ++r, dst += a.out_pitch) {
                const int q[4] = {q4.x, q4.y, q4.z, q4.w};
                q4 = e[r + 1];
#pragma unroll
                for (int i = 0; i < 2 * S2; ++i)
                    if (q[i] & 1) load_row<K2>(v[i], lane_base + (q[i] - 1));
                float o[K2];
                add_rows<K2>(o, v[0], v[1]);
                if constexpr (S2 == 2) {
                    float h[K2];
                    add_rows<K2>(h, v[2], v[3]);
                    add_rows<K2>(o, o, h);
                }
                if (clean) {
#pragma unroll
                    for (int k = 0; k < K2; ++k) dst[32 * k] = o[k];
                } else {
                    const int lim = a.ncols - t0 - lane;   // samples left from this lane's first
#pragma unroll
                    for (int k = 0; k < K2; ++k)
                        if (32 * k < lim) dst[32 * k] = o[k];
                }
            }
        }
        t = next;
        rt = rn;
        tt = tn;
    }
}

template <int S1, int S2, int R0C, bool POS>
cudaError_t launch(const RunPlan& rp, const RunArgs& args, cudaStream_t s) {
    auto kern = k_fdmt_run<S1, S2, R0C, POS>;
    // The shared-memory opt-in (one value per kernel and device, it only ever
    // grows) and the resident CTAs of a size are set on the size's first
    // launch, which therefore comes before any stream capture.
    static std::mutex mu;
    static std::map<int, size_t> optin;
    static std::map<std::pair<int, size_t>, int> resident;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int ctas = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        size_t& have = optin[dev];
        if (have < rp.smem_bytes) {
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(rp.smem_bytes));
            if (e != cudaSuccess) return e;
            have = rp.smem_bytes;
        }
        auto it = resident.find({dev, rp.smem_bytes});
        if (it == resident.end()) {
            int per_sm = 0, sms = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kRunThreads, rp.smem_bytes);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            if (per_sm < 1) return cudaErrorInvalidConfiguration;
            it = resident.emplace(std::make_pair(dev, rp.smem_bytes), per_sm * sms).first;
        }
        ctas = it->second;
    }
    kern<<<std::min(args.total, ctas), kRunThreads, rp.smem_bytes, s>>>(args);
    return cudaGetLastError();
}

template <int R0C, bool POS = false>
cudaError_t launch_stages(const RunPlan& rp, const RunArgs& a, cudaStream_t s) {
    if (rp.s1 == 2 && rp.s2 == 2) return launch<2, 2, R0C, POS>(rp, a, s);
    if (rp.s1 == 2 && rp.s2 == 1) return launch<2, 1, R0C, POS>(rp, a, s);
    if (rp.s1 == 1 && rp.s2 == 1) return launch<1, 1, R0C, POS>(rp, a, s);
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_run(const RunPlan& rp, const float* src, float* dst, const RunTile* tiles, const int2* rows,
                       const int4* ent, int ncols, int in_pitch, int out_pitch, int ones, cudaStream_t s) {
    RunArgs a;
    a.in = src; a.out = dst; a.tiles = tiles; a.rows = rows; a.ent = ent;
    a.ncols = ncols; a.in_pitch = in_pitch; a.out_pitch = out_pitch;
    a.nrt = static_cast<int>(rp.tiles.size());
    const long long total = static_cast<long long>(a.nrt) * ((ncols + kSegTile - 1) / kSegTile);
    if (total > (1LL << 30)) return cudaErrorInvalidConfiguration;
    a.total = static_cast<int>(total);
    a.pitch_x = rp.pitch_x; a.zero_x = rp.zero_x; a.zero_y = rp.zero_y; a.y0 = rp.y0;
    a.ent0 = rp.ent0; a.max_ent = rp.max_ent; a.edge = rp.edge;
    // planes have a pitch of whole 16-byte pieces; a channel's window starts
    // on a 16-byte boundary when the filterbank does
    a.vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && (rp.r0c > 0 || in_pitch % 4 == 0) ? 1 : 0;
    a.ones = ones;
    if (rp.positive) return launch_stages<5, true>(rp, a, s);
    switch (rp.r0c) {
        case 0: case 1: return launch_stages<0>(rp, a, s);
        case 2: return launch_stages<2>(rp, a, s);
        case 3: return launch_stages<3>(rp, a, s);
        case 4: return launch_stages<4>(rp, a, s);
        case 5: return launch_stages<5>(rp, a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bfs
