// Run segments over 16-bit planes (sm_100a): the passes of fdmt_run.cu with
// FP16 or BF16 values in HBM, in shared memory and in registers.  A plain
// 16-bit level stores rn16(rn32(a 2^l + b 2^l) 2^-(l+1)); where every row of
// level l has the scale 2^-l that is rn16(a + b) / 2 for the stored a and b:
// a sum rounded to FP32 and then to 16 bits equals the sum rounded once (24 >=
// 2 p + 2 bits), and the halving of it is exact or rounds an exact sum.  Only a
// sum beyond the type's range differs; a warp that meets one forms its rows
// again as the plain level forms them.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "fdmt_run.h"
#include "row_ops.cuh"

namespace bfs {
namespace {

constexpr int kThreads16 = 256;
constexpr int kWarps16 = kThreads16 / 32;
constexpr int kMidWords = kRun16Mid / 64, kOutWords = kRun16Tile / 64;

template <typename S> struct Pair;
template <> struct Pair<__half> {
    using V = __half2;
    static __device__ __forceinline__ float wide(unsigned short v) { return __half2float(__ushort_as_half(v)); }
    static __device__ __forceinline__ unsigned short narrow(float v) { return __half_as_ushort(__float2half_rn(v)); }
    static __device__ __forceinline__ float2 wide2(V v) { return __half22float2(v); }
    static __device__ __forceinline__ V half() { return __floats2half2_rn(0.5f, 0.5f); }
    // a sum that overflowed leaves an infinity or a NaN, and 0 times either is NaN
    static __device__ __forceinline__ V track(V worst, V o) { return __hfma2(o, __floats2half2_rn(0.0f, 0.0f), worst); }
    static __device__ __forceinline__ bool in_range(V worst) { return __hbeq2(worst, worst); }
};
template <> struct Pair<__nv_bfloat16> {
    using V = __nv_bfloat162;
    static __device__ __forceinline__ float wide(unsigned short v) { return __bfloat162float(__ushort_as_bfloat16(v)); }
    static __device__ __forceinline__ unsigned short narrow(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }
    static __device__ __forceinline__ float2 wide2(V v) { return __bfloat1622float2(v); }
    static __device__ __forceinline__ V half() { return __floats2bfloat162_rn(0.5f, 0.5f); }
    // (up to 2^100 the scaled-up value of any level is a finite float, too)
    static __device__ __forceinline__ V track(V worst, V o) { return __hmax2_nan(worst, __habs2(o)); }
    static __device__ __forceinline__ bool in_range(V worst) { return __hble2(worst, __floats2bfloat162_rn(0x1p100f, 0x1p100f)); }
};

__device__ __forceinline__ float exp2_int16(int e) { return __int_as_float((127 + e) << 23); }

struct Run16Args {
    const void* in;
    void* out;
    const RunTile* tiles;
    const int2* rows;
    const int4* ent;
    int ncols, in_pitch, out_pitch, nrt, total;
    int pitch_x, zero_x, zero_y, y0, ent0, max_ent;   // values (2 bytes each)
    int level;                                        // l0
    int vec;                                          // FP32 output rows start on 8-byte boundaries
};

// Word k of a lane: columns 64 k + 2 lane and the next, from byte offset q
// (bit 0: the row's moved flag; bit 1: an odd sample, two words and a cut).
template <int K>
__device__ __forceinline__ void load16(unsigned (&v)[K], const char* lane_base, int q) {
    const char* p = lane_base + (q & ~3);
    if (q & 2) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            v[k] = __byte_perm(*reinterpret_cast<const unsigned*>(p + 128 * k),
                               *reinterpret_cast<const unsigned*>(p + 128 * k + 4), 0x5432);
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = *reinterpret_cast<const unsigned*>(p + 128 * k);
    }
}

template <typename S>
__device__ __forceinline__ typename Pair<S>::V pair_of(const unsigned& w) {
    return *reinterpret_cast<const typename Pair<S>::V*>(&w);
}

// rn16(a + b) / 2, in pairs.
template <typename S>
__device__ __forceinline__ unsigned merge16(unsigned a, unsigned b) {
    const typename Pair<S>::V o = __hmul2_rn(__hadd2_rn(pair_of<S>(a), pair_of<S>(b)), Pair<S>::half());
    return *reinterpret_cast<const unsigned*>(&o);
}

// One value of a row as the plain levels form it, before its last store; the
// inputs are level-l values at byte offsets q of shared memory, column col.
template <typename S, int LEVELS>
__device__ __noinline__ float plain16(const char* sm, int4 q, int col, int l) {
    auto at = [&](int e) {
        return __fmul_rn(Pair<S>::wide(*reinterpret_cast<const unsigned short*>(sm + (e & ~1) + 2 * col)), exp2_int16(l));
    };
    const float v = __fadd_rn(at(q.x), at(q.y));
    if (LEVELS == 1) return v;
    const float h = __fadd_rn(at(q.z), at(q.w));
    auto stored = [&](float x) {
        return __fmul_rn(Pair<S>::wide(Pair<S>::narrow(__fmul_rn(x, exp2_int16(-l - 1)))), exp2_int16(l + 1));
    };
    return __fadd_rn(stored(v), stored(h));
}

// The shape of the loops is k_fdmt_run's.  A lane holds two neighbouring
// columns, so that an input at an even offset costs one shared wavefront per 64
// columns, at an odd one two and a cut.  Bound by instruction issue (59-63 % of
// the slots at 16 warps per SM) and the dependent latencies between them: 4096 x
// 131072, levels 1..12 in three passes of four: 2.39 ms; one plain pass per level
// 5.9 ms.  Slower: tiles of 256 samples at three CTAs per SM (a row's fixed
// instructions are as many as its merges), four CTAs (spills), the range tested
// row by row.
template <typename S, int S1, int S2, bool F32OUT>
__global__ void __launch_bounds__(kThreads16, 2) k_fdmt_run16(const Run16Args a) {
    using V = typename Pair<S>::V;
    constexpr int K1 = kMidWords, K2 = kOutWords;
    extern __shared__ __align__(16) char sm16[];
    unsigned* words = reinterpret_cast<unsigned*>(sm16);
    const unsigned sbase = static_cast<unsigned>(__cvta_generic_to_shared(sm16));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const char* lane_base = sm16 + 4 * lane;
    constexpr unsigned kNegZero = 0x80008000u;
    for (int i = threadIdx.x; i < kRun16Mid / 2; i += kThreads16) words[a.zero_x / 2 + i] = kNegZero;
    for (int i = threadIdx.x; i < kRun16Tile / 2; i += kThreads16) words[a.zero_y / 2 + i] = kNegZero;

    auto tile_of = [&](int rt) {
        const int4* p = reinterpret_cast<const int4*>(a.tiles + rt);
        const int4 lo = __ldg(p), hi = __ldg(p + 1);
        RunTile t{};
        t.row = lo.x; t.ent = lo.y; t.n_in = lo.z; t.n1 = lo.w; t.n2 = hi.x; t.out0 = hi.y;
        return t;
    };
    auto row_entries = [&](const RunTile& t) {
        const int j = warp + kWarps16 * lane;
        return j < t.n_in ? __ldg(a.rows + t.row + j) : make_int2(0, 0);
    };
    auto issue = [&](const RunTile& t, int2 mine, int tt, int eb) {
        const int nent = t.n1 + t.n2;
        const unsigned se = sbase + 2u * a.ent0 + 16u * eb * a.max_ent;
        for (int i = threadIdx.x; i < nent; i += kThreads16) copy16(se + 16u * i, a.ent + t.ent + i);
        const int t0 = tt * kRun16Tile;
        const int pieces = a.pitch_x >> 3;
        // the last row's reads run past its end, into a row that this tile does
        // not load: what lies there would decide whether sums left the range
        if (threadIdx.x < kRun16Over / 8 && t.n_in * a.pitch_x < a.zero_x)
            *reinterpret_cast<uint4*>(sm16 + 2 * (t.n_in * a.pitch_x) + 16 * threadIdx.x) = make_uint4(0u, 0u, 0u, 0u);
        for (int i = 0, j = warp; j < t.n_in; ++i, j += kWarps16) {
            const int row = __shfl_sync(0xffffffffu, mine.x, i), lead = __shfl_sync(0xffffffffu, mine.y, i);
            const int ts = t0 - lead;   // a multiple of 8: a piece lies before sample 0 or from it on
            const S* src = static_cast<const S*>(a.in) + static_cast<size_t>(row) * a.in_pitch + ts;
            const unsigned dst = sbase + 2u * (j * a.pitch_x);
            if (ts >= 0 && ts + a.pitch_x <= a.ncols) {
                for (int c = lane; c < pieces; c += 32) copy16(dst + 16u * c, src + 8 * c);
                continue;
            }
            for (int c = lane; c < pieces; c += 32) {
                const int at = ts + 8 * c;
                if (at >= 0 && at + 8 <= a.ncols) {
                    copy16(dst + 16u * c, src + 8 * c);
                    continue;
                }
                uint4 v = at < 0 ? make_uint4(kNegZero, kNegZero, kNegZero, kNegZero) : make_uint4(0u, 0u, 0u, 0u);
                if (at >= 0 && at < a.ncols) {   // the row's end: what lies past it may never have been written
                    const int left = a.ncols - at;
                    auto cut = [&](unsigned w, int first) { return left > first + 1 ? w : left > first ? w & 0xffffu : 0u; };
                    v = *reinterpret_cast<const uint4*>(src + 8 * c);
                    v = make_uint4(cut(v.x, 0), cut(v.y, 2), cut(v.z, 4), cut(v.w, 6));
                }
                *reinterpret_cast<uint4*>(sm16 + 2 * (j * a.pitch_x) + 16 * c) = v;
            }
        }
    };

    const int G = static_cast<int>(gridDim.x);
    const int gq = G / a.nrt, gr = G % a.nrt;
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
        const int t0 = tt * kRun16Tile;
        const int4* e = reinterpret_cast<const int4*>(sm16 + 2 * a.ent0) + eb * a.max_ent;
        {
            const int r0 = t.n1 * warp / kWarps16, r1 = t.n1 * (warp + 1) / kWarps16;
            unsigned* dst = words + (a.y0 + r0 * kRun16Mid) / 2 + lane;
            unsigned v[2 * S1][K1];
            V worst = pair_of<S>(0u);
            int4 q4 = e[r0];
            q4 = make_int4(q4.x | 1, q4.y | 1, q4.z | 1, q4.w | 1);   // a warp's first row reads all its inputs
#pragma unroll 1
            for (int r = r0; r < r1; ++r, dst += kRun16Mid / 2) {
                const int q[4] = {q4.x, q4.y, q4.z, q4.w};
                q4 = e[r + 1];
#pragma unroll
                for (int i = 0; i < 2 * S1; ++i)
                    if (q[i] & 1) load16<K1>(v[i], lane_base, q[i]);
#pragma unroll
                for (int k = 0; k < K1; ++k) {
                    unsigned o = merge16<S>(v[0][k], v[1][k]);
                    if constexpr (S1 == 2) o = merge16<S>(o, merge16<S>(v[2][k], v[3][k]));
                    worst = Pair<S>::track(worst, pair_of<S>(o));
                    dst[32 * k] = o;
                }
            }
            if (!__all_sync(0xffffffffu, Pair<S>::in_range(worst))) {
                __syncwarp();   // the stores above come first
                for (int r = r0; r < r1; ++r)
                    for (int col = lane; col < kRun16Mid; col += 32)
                        reinterpret_cast<unsigned short*>(sm16)[a.y0 + r * kRun16Mid + col] = Pair<S>::narrow(
                            __fmul_rn(plain16<S, S1>(sm16, e[r], col, a.level), exp2_int16(-a.level - S1)));
            }
        }
        __syncthreads();   // Y is in, every warp is done with X
        if (more) issue(next, next_rows, tn, eb ^ 1);
        {
            e += t.n1;
            const int l = a.level + S1;
            const int r0 = t.n2 * warp / kWarps16, r1 = t.n2 * (warp + 1) / kWarps16;
            const int c0 = t0 + 2 * lane;
            unsigned v[2 * S2][K2];
            V worst = pair_of<S>(0u);
            int4 q4 = e[r0];
            q4 = make_int4(q4.x | 1, q4.y | 1, q4.z | 1, q4.w | 1);
#pragma unroll 1
            for (int r = r0; r < r1; ++r) {
                const int q[4] = {q4.x, q4.y, q4.z, q4.w};
                q4 = e[r + 1];
#pragma unroll
                for (int i = 0; i < 2 * S2; ++i)
                    if (q[i] & 1) load16<K2>(v[i], lane_base, q[i]);
                const size_t row = static_cast<size_t>(t.out0 + r) * a.out_pitch;
                if constexpr (F32OUT) {
                    float* out = static_cast<float*>(a.out) + row + c0;
                    const float scale = exp2_int16(l + S2 - 1);
#pragma unroll
                    for (int k = 0; k < K2; ++k) {
                        unsigned x = v[0][k], y = v[1][k];
                        if constexpr (S2 == 2) {
                            x = merge16<S>(v[0][k], v[1][k]);
                            y = merge16<S>(v[2][k], v[3][k]);
                            worst = Pair<S>::track(Pair<S>::track(worst, pair_of<S>(x)), pair_of<S>(y));
                        }
                        const float2 fx = Pair<S>::wide2(pair_of<S>(x)), fy = Pair<S>::wide2(pair_of<S>(y));
                        const float o0 = __fadd_rn(__fmul_rn(fx.x, scale), __fmul_rn(fy.x, scale));
                        const float o1 = __fadd_rn(__fmul_rn(fx.y, scale), __fmul_rn(fy.y, scale));
                        const int c = c0 + 64 * k;
                        if (a.vec && c + 1 < a.ncols) {
                            *reinterpret_cast<float2*>(out + 64 * k) = make_float2(o0, o1);
                        } else {
                            if (c < a.ncols) out[64 * k] = o0;
                            if (c + 1 < a.ncols) out[64 * k + 1] = o1;
                        }
                    }
                } else {
                    // (rows have whole 128-byte lines: a word past ncols is the row's own)
                    unsigned* out = reinterpret_cast<unsigned*>(static_cast<S*>(a.out) + row) + c0 / 2;
#pragma unroll
                    for (int k = 0; k < K2; ++k) {
                        unsigned o = merge16<S>(v[0][k], v[1][k]);
                        if constexpr (S2 == 2) o = merge16<S>(o, merge16<S>(v[2][k], v[3][k]));
                        worst = Pair<S>::track(worst, pair_of<S>(o));
                        if (c0 + 64 * k < a.ncols) out[32 * k] = o;
                    }
                }
            }
            if (!__all_sync(0xffffffffu, Pair<S>::in_range(worst))) {
                __syncwarp();   // the stores above come first
                for (int r = r0; r < r1; ++r)
                    for (int col = lane; col < kRun16Tile && t0 + col < a.ncols; col += 32) {
                        const float o = plain16<S, S2>(sm16, e[r], col, l);
                        const size_t at = static_cast<size_t>(t.out0 + r) * a.out_pitch + t0 + col;
                        if constexpr (F32OUT) static_cast<float*>(a.out)[at] = o;
                        else static_cast<unsigned short*>(a.out)[at] = Pair<S>::narrow(__fmul_rn(o, exp2_int16(-l - S2)));
                    }
            }
        }
        t = next;
        rt = rn;
        tt = tn;
    }
}

template <typename S, int S1, int S2, bool F32OUT>
cudaError_t launch16(const RunPlan& rp, const Run16Args& args, cudaStream_t s) {
    auto kern = k_fdmt_run16<S, S1, S2, F32OUT>;
    // The opt-in and the resident CTAs of a size: as for k_fdmt_run, set on a
    // size's first launch, which comes before any stream capture.
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
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads16, rp.smem_bytes);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            if (per_sm < 1) return cudaErrorInvalidConfiguration;
            it = resident.emplace(std::make_pair(dev, rp.smem_bytes), per_sm * sms).first;
        }
        ctas = it->second;
    }
    kern<<<std::min(args.total, ctas), kThreads16, rp.smem_bytes, s>>>(args);
    return cudaGetLastError();
}

template <typename S, bool F32OUT>
cudaError_t launch_stages16(const RunPlan& rp, const Run16Args& a, cudaStream_t s) {
    if (rp.s1 == 2 && rp.s2 == 2) return launch16<S, 2, 2, F32OUT>(rp, a, s);
    if (rp.s1 == 2 && rp.s2 == 1) return launch16<S, 2, 1, F32OUT>(rp, a, s);
    if (rp.s1 == 1 && rp.s2 == 1) return launch16<S, 1, 1, F32OUT>(rp, a, s);
    return cudaErrorInvalidValue;
}

}  // namespace

template <typename S>
cudaError_t launch_run16(const RunPlan& rp, const S* src, void* dst, bool out_f32, const RunTile* tiles,
                         const int2* rows, const int4* ent, int ncols, int in_pitch, int out_pitch, cudaStream_t s) {
    Run16Args a;
    a.in = src; a.out = dst; a.tiles = tiles; a.rows = rows; a.ent = ent;
    a.ncols = ncols; a.in_pitch = in_pitch; a.out_pitch = out_pitch;
    a.nrt = static_cast<int>(rp.tiles.size());
    const long long total = static_cast<long long>(a.nrt) * ((ncols + kRun16Tile - 1) / kRun16Tile);
    if (total > (1LL << 30)) return cudaErrorInvalidConfiguration;
    a.total = static_cast<int>(total);
    a.pitch_x = rp.pitch_x; a.zero_x = rp.zero_x; a.zero_y = rp.zero_y; a.y0 = rp.y0;
    a.ent0 = rp.ent0; a.max_ent = rp.max_ent;
    a.level = rp.l0;
    a.vec = out_f32 && out_pitch % 2 == 0 && reinterpret_cast<uintptr_t>(dst) % 8 == 0 ? 1 : 0;
    return out_f32 ? launch_stages16<S, true>(rp, a, s) : launch_stages16<S, false>(rp, a, s);
}

template cudaError_t launch_run16<__half>(const RunPlan&, const __half*, void*, bool, const RunTile*, const int2*,
                                          const int4*, int, int, int, cudaStream_t);
template cudaError_t launch_run16<__nv_bfloat16>(const RunPlan&, const __nv_bfloat16*, void*, bool, const RunTile*,
                                                 const int2*, const int4*, int, int, int, cudaStream_t);

}  // namespace bfs
