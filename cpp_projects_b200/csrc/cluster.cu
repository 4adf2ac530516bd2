// Candidate clustering and delegate selection on sm_100a.
//
// Reference: clusterization::complete_clusterization
// (L/Clusterization/Clusterization.cu:92-166) runs three grouping passes over
// the candidate fields mt, mdt and mwidth.  Each pass sorts the members of
// every current group by the field (sort_subarrays_cub_,
// L/Clusterization/Segmented_sort.cu:87-124) and starts a new group wherever
// two consecutive values differ by more than the pass's metric
// (calc_plan_and_values_for_regrouping_kernel / regrouping_kernel,
// Clusterization.cu:855-998).  A delegate is then picked per group
// (select_delegates_kernel, L/Clusterization/select_delegates.cu:63-125) and
// the delegates are sorted by mt (Clusterization.cu:147-149).
//
// Here one pass is: 64-bit key (group id << 32 | biased field value), a
// stable device radix sort of (key, candidate index) in index order — so ties
// resolve by candidate index, deterministically — a split-flag kernel, an
// inclusive scan of the flags (new group ids) and a scatter of the new ids.
// Where the passes' (group, field) cells are few enough for a bitmap, no pass
// sorts: the group numbers come from the bitmap's gaps and one sort by (group,
// width) gives the member order (cluster_by_gaps).
// The reference's segmented sort is unstable; the group SETS it produces are
// the same (splits depend only on the sorted values), only the order inside
// a group differs, and the canonical order here is by candidate index.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <cfloat>
#include <climits>

#include "internal.h"

namespace bfs {
namespace {

constexpr int kDelegateLanes = 64;  // select_delegates_kernel's block size in the reference

__device__ __forceinline__ int field_of(const bfs_cand& c, int f) {
    return f == 0 ? c.mt : (f == 1 ? c.mdt : c.mwidth);
}

__device__ __forceinline__ unsigned biased(int v) { return static_cast<unsigned>(v) ^ 0x80000000u; }

// Pass key: (group id << fbits) | (field - fmin), in 32 bits when it fits.
template <typename K>
__global__ void k_pass_keys(const bfs_cand* __restrict__ c, const unsigned* __restrict__ gid,
                            unsigned n, int field, int fmin, int fbits, K* __restrict__ keys,
                            unsigned* __restrict__ vals) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const K g = gid ? static_cast<K>(gid[i]) : K(0);
    const K f = static_cast<K>(static_cast<unsigned>(
        static_cast<long long>(field_of(c[i], field)) - static_cast<long long>(fmin)));
    keys[i] = (fbits >= static_cast<int>(8 * sizeof(K)) ? K(0) : (g << fbits)) | f;
    vals[i] = i;
}

// Group starts in the sorted order: the group changes, or the field grows by
// more than the metric.  A key's low fbits bits are its field minus the
// smallest field (exact: fbits covers the range), so the sorted keys alone
// give both tests.
template <typename K>
__global__ void k_pass_flags(const K* __restrict__ keys, unsigned n, int fbits, long long metric,
                             unsigned* __restrict__ flags) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned f = 1u;
    if (i > 0) {
        const bool whole = fbits >= static_cast<int>(8 * sizeof(K));
        const K k0 = keys[i - 1], k1 = keys[i];
        const K g0 = whole ? K(0) : (k0 >> fbits);
        const K g1 = whole ? K(0) : (k1 >> fbits);
        if (g0 == g1) {
            const K mask = whole ? ~K(0) : ((K(1) << fbits) - K(1));
            const long long d = static_cast<long long>(k1 & mask) - static_cast<long long>(k0 & mask);
            f = (d > metric) ? 1u : 0u;
        }
    }
    flags[i] = f;
}

// Range of each field (biased so signed order is unsigned order), as the
// complement of the smallest and the largest, both maxima over zeros; then the
// largest initial group (as unsigned).  One
// atomic per CTA and bound: 38.9 us with one per warp at 0.3 M candidates.
constexpr int kRangeThreads = 512, kRanges = 7;
__global__ void __launch_bounds__(kRangeThreads)
k_field_range(const bfs_cand* __restrict__ c, const int* __restrict__ g0, unsigned n, unsigned* __restrict__ r) {
    __shared__ unsigned sh[kRanges];
    if (threadIdx.x < kRanges) sh[threadIdx.x] = 0u;
    __syncthreads();
    unsigned m[kRanges] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const bfs_cand v = c[i];
        const unsigned f[3] = {biased(v.mt), biased(v.mdt), biased(v.mwidth)};
        for (int k = 0; k < 3; ++k) { m[2 * k] = max(m[2 * k], ~f[k]); m[2 * k + 1] = max(m[2 * k + 1], f[k]); }
        if (g0) m[6] = max(m[6], static_cast<unsigned>(__ldg(g0 + i)));
    }
    for (int k = 0; k < kRanges; ++k) {
        const unsigned v = __reduce_max_sync(0xffffffffu, m[k]);
        if ((threadIdx.x & 31) == 0) atomicMax(sh + k, v);
    }
    __syncthreads();
    if (threadIdx.x < kRanges) atomicMax(r + threadIdx.x, sh[threadIdx.x]);
}

__global__ void k_pass_scatter(const unsigned* __restrict__ vals, const unsigned* __restrict__ scan,
                               unsigned n, unsigned* __restrict__ gid) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) gid[vals[i]] = scan[i] - 1u;
}

__global__ void k_offsets(const unsigned* __restrict__ flags, const unsigned* __restrict__ scan,
                          unsigned n, int* __restrict__ offsets) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && flags[i]) offsets[scan[i] - 1u] = static_cast<int>(i);
    if (i == n - 1) offsets[scan[i]] = static_cast<int>(n);
}

// Delegate selection, exactly the reference's select_delegates_kernel
// (64 lanes per group; lane l keeps the first strict maximum of msnr among the
// group positions l, l+64, ...; a tree reduction `take lane l+s if strictly
// greater` for s = 32..1) but split in two so that groups of millions of
// members do not serialise on 64 threads:
//   k_delegate_lanes  every position of every group, 16 or 4 per thread (stride 64,
//                     so a thread stays on one lane of a group) keeps the
//                     largest key (ordered msnr << 32 | ~position) and folds it
//                     into its (group, lane) slot with a 64-bit atomicMax:
//                     the largest value, earliest position on ties = the
//                     reference lane's strided scan;
//   k_delegate_tree   one 64-thread block per group runs the reference's tree.
constexpr int kLaneThreads = 256;

__device__ __forceinline__ unsigned ordered_bits(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ int group_of(const int* __restrict__ offsets, int ngroups, int i) {
    int lo = 0, hi = ngroups - 1;  // largest g with offsets[g] <= i
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(offsets + mid) <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

template <int kLanePositions>
__global__ void __launch_bounds__(kLaneThreads)
k_delegate_lanes(const bfs_cand* __restrict__ c, const int* __restrict__ perm, int n,
                 const int* __restrict__ offsets, int ngroups,
                 unsigned long long* __restrict__ slots) {
    const int sub = threadIdx.x / kDelegateLanes, lane = threadIdx.x % kDelegateLanes;
    const int base = blockIdx.x * (kLaneThreads * kLanePositions) + sub * (kDelegateLanes * kLanePositions) + lane;
    int g = -1, g_beg = 0, g_end = 0;
    unsigned long long best = 0ull;
    for (int k = 0; k < kLanePositions; ++k) {
        const int i = base + k * kDelegateLanes;
        if (i >= n) break;
        if (g < 0 || i >= g_end) {
            if (best) atomicMax(slots + static_cast<size_t>(g) * kDelegateLanes + ((base - g_beg) & 63), best);
            g = group_of(offsets, ngroups, i);
            g_beg = __ldg(offsets + g);
            g_end = __ldg(offsets + g + 1);
            best = 0ull;
        }
        const unsigned pos = static_cast<unsigned>(i - g_beg);
        const unsigned long long key =
            (static_cast<unsigned long long>(ordered_bits(c[__ldg(perm + i)].msnr)) << 32) |
            static_cast<unsigned long long>(0xffffffffu - pos);
        best = key > best ? key : best;
    }
    if (best) atomicMax(slots + static_cast<size_t>(g) * kDelegateLanes + ((base - g_beg) & 63), best);
}

__global__ void __launch_bounds__(kDelegateLanes)
k_delegate_tree(const bfs_cand* __restrict__ c, const int* __restrict__ perm,
                const int* __restrict__ offsets, const unsigned long long* __restrict__ slots,
                int* __restrict__ delegates) {
    __shared__ float sv[kDelegateLanes];
    __shared__ int si[kDelegateLanes];
    const int g = blockIdx.x;
    const int beg = offsets[g];
    const int len = offsets[g + 1] - beg;
    const int lane = threadIdx.x;
    float v = -FLT_MAX;
    int idx = lane;  // the reference leaves the lane id in idle lanes
    if (lane < len) {
        const unsigned long long key = slots[static_cast<size_t>(g) * kDelegateLanes + lane];
        const unsigned pos = 0xffffffffu - static_cast<unsigned>(key & 0xffffffffull);
        idx = perm[beg + pos];
        v = c[idx].msnr;
    }
    sv[lane] = v;
    si[lane] = idx;
    __syncthreads();
    for (int s = kDelegateLanes / 2; s > 0; s >>= 1) {
        if (lane < s && sv[lane + s] > sv[lane]) { sv[lane] = sv[lane + s]; si[lane] = si[lane + s]; }
        __syncthreads();
    }
    if (lane == 0) delegates[g] = si[0];
}

bfs_status launch_select_delegates(const bfs_cand* c, const int* perm, unsigned n,
                                   const int* offsets, unsigned ngroups, int* out,
                                   unsigned long long* slots, cudaStream_t s) {
    if (ngroups == 0) return BFS_OK;
    BFS_CUDA(cudaMemsetAsync(slots, 0, sizeof(unsigned long long) * kDelegateLanes * ngroups, s));
    // a thread's positions are a chain of dependent loads: few of them until
    // the blocks fill the chip (0.3 M candidates: 19.5 us with 16)
    auto blocks = [&](unsigned per) { return (n + kLaneThreads * per - 1) / (kLaneThreads * per); };
    if (blocks(16) >= 2 * 148)
        k_delegate_lanes<16><<<blocks(16), kLaneThreads, 0, s>>>(c, perm, static_cast<int>(n), offsets,
                                                                 static_cast<int>(ngroups), slots);
    else
        k_delegate_lanes<4><<<blocks(4), kLaneThreads, 0, s>>>(c, perm, static_cast<int>(n), offsets,
                                                               static_cast<int>(ngroups), slots);
    BFS_LAUNCH_CHECK("k_delegate_lanes");
    k_delegate_tree<<<ngroups, kDelegateLanes, 0, s>>>(c, perm, offsets, slots, out);
    BFS_LAUNCH_CHECK("k_delegate_tree");
    return BFS_OK;
}

// (delegates are given in group order and the sort is stable, so mt alone,
// less the smallest, orders them by (mt, group))
__global__ void k_delegate_keys(const bfs_cand* __restrict__ c, const int* __restrict__ dl, unsigned ng, int tmin,
                                unsigned* __restrict__ keys, unsigned* __restrict__ vals) {
    const unsigned g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    keys[g] = static_cast<unsigned>(c[dl[g]].mt) - static_cast<unsigned>(tmin);
    vals[g] = static_cast<unsigned>(dl[g]);
}

// ---- grouping by gaps ----------------------------------------------------------
// A pass numbers its groups in the order of (group, field); a new one starts
// at a field value whose predecessor in the group is more than the metric
// below it.  So the pass needs the set of (group, field) cells in use, not the
// members' order: cell p = (group << shift) + field - fmin marks bit p of a
// bitmap, and a member's new group is the number of starts at bits <= p, less
// one.  A scan over the bitmap's words carries {first, last bit, starts after
// the first}; per word it leaves its starts and the starts before it.
struct GapState { unsigned first, last, n, any; };

struct GapRule {
    int shift;
    unsigned metric;
    __device__ bool split(unsigned p, unsigned q) const {   // p < q: neighbouring cells in use
        return (p >> shift) != (q >> shift) || q - p > metric;
    }
    __device__ GapState operator()(const GapState& a, const GapState& b) const {
        if (!a.any) return b;
        if (!b.any) return a;
        return GapState{a.first, b.last, a.n + b.n + (split(a.last, b.first) ? 1u : 0u), 1u};
    }
};

// bits of a word whose predecessor inside the word is more than the metric
// below (the lowest set bit always is one); groups are whole words
__device__ __forceinline__ unsigned word_starts(unsigned bits, unsigned metric) {
    unsigned near = 0u;
    for (unsigned k = 1; k <= metric && k < 32u; ++k) near |= bits << k;
    return bits & ~near;
}

struct GapWord {
    const unsigned* bits;
    unsigned metric;
    __device__ GapState operator()(unsigned w) const {
        const unsigned b = bits[w];
        if (!b) return GapState{0u, 0u, 0u, 0u};
        return GapState{32u * w + __ffs(b) - 1u, 32u * w + 31u - __clz(b),
                        static_cast<unsigned>(__popc(word_starts(b, metric))) - 1u, 1u};
    }
};

// tab[w] = {starts of word w, starts before it}; *total = groups
__global__ void k_gap_table(const unsigned* __restrict__ bits, const GapState* __restrict__ before, unsigned words,
                            GapRule rule, uint2* __restrict__ tab, unsigned* __restrict__ total) {
    const unsigned w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= words) return;
    const unsigned b = bits[w];
    const GapState p = before[w];
    unsigned s = word_starts(b, rule.metric);
    if (b && p.any && !rule.split(p.last, 32u * w + __ffs(b) - 1u)) s &= s - 1u;   // the first goes on from before
    const unsigned base = p.any ? p.n + 1u : 0u;
    tab[w] = make_uint2(s, base);
    if (w == words - 1) *total = base + __popc(s);
}

struct GapMap {          // a pass's table (null: the pass cannot split)
    const uint2* tab;
    int fmin, shift;
};

__device__ __forceinline__ unsigned gap_cell(const bfs_cand& c, int field, unsigned g, int fmin, int shift) {
    return (g << shift) + (static_cast<unsigned>(field_of(c, field)) - static_cast<unsigned>(fmin));
}

// group of a member after the first `passes` of the maps
__device__ __forceinline__ unsigned gap_group(const bfs_cand& c, unsigned g, const GapMap (&m)[3], int passes) {
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        if (f >= passes || !m[f].tab) continue;
        const unsigned p = gap_cell(c, f, g, m[f].fmin, m[f].shift);
        const uint2 t = __ldg(m[f].tab + (p >> 5));
        g = t.y + __popc(t.x & ((2u << (p & 31u)) - 1u)) - 1u;
    }
    return g;
}

struct GapMaps { GapMap m[3]; };

// Marks the cells of a CTA's contiguous share of the candidates.  Neighbours
// lie in few words and the words of a bright pulse are hit by most of the
// list, so a warp sets a word's bits with one atomic, and only where a small
// table of the words this CTA has set does not hold them yet (with a look at
// the word in L2 instead the hot words' lines were the bound: 126 us for 4 M
// candidates, 13 us for 0.3 M).
constexpr int kMarkCache = 1024;
__global__ void __launch_bounds__(256)
k_gap_mark(const bfs_cand* __restrict__ c, const int* __restrict__ g0, unsigned n, unsigned per_cta, GapMaps maps,
           int field, int fmin, int shift, unsigned words, unsigned* __restrict__ bits) {
    __shared__ unsigned long long known[kMarkCache];   // {word + 1, its bits}: one 8-byte access each
    for (int i = threadIdx.x; i < kMarkCache; i += blockDim.x) known[i] = 0ull;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const unsigned beg = blockIdx.x * per_cta, end = min(n, beg + per_cta);
    for (unsigned i0 = beg; i0 < end; i0 += blockDim.x) {   // CTA-uniform
        const unsigned i = i0 + threadIdx.x;
        unsigned w = 0xffffffffu, b = 0u;
        if (i < end) {
            const bfs_cand v = c[i];
            const unsigned p =
                gap_cell(v, field, gap_group(v, g0 ? static_cast<unsigned>(__ldg(g0 + i)) : 0u, maps.m, field), fmin, shift);
            w = p >> 5;
            b = 1u << (p & 31u);
        }
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {   // the lane's bits and those of the lanes after it in the same word
            const unsigned uw = __shfl_down_sync(0xffffffffu, w, d), ub = __shfl_down_sync(0xffffffffu, b, d);
            if (lane + d < 32 && uw == w) b |= ub;
        }
        const unsigned left = __shfl_up_sync(0xffffffffu, w, 1);
        if (w >= words || (lane != 0 && left == w)) continue;
        const unsigned long long k = *const_cast<volatile unsigned long long*>(known + (w & (kMarkCache - 1)));
        if ((k >> 32) == w + 1ull && (static_cast<unsigned>(k) & b) == b) continue;
        const unsigned old = atomicOr(bits + w, b);
        *const_cast<volatile unsigned long long*>(known + (w & (kMarkCache - 1))) = (w + 1ull) << 32 | (old | b);
    }
}

// keys of the final order: (group, width), ties by index
template <typename K>
__global__ void k_gap_keys(const bfs_cand* __restrict__ c, const int* __restrict__ g0, unsigned n, GapMaps maps,
                           int wmin, int wbits, K* __restrict__ keys, unsigned* __restrict__ vals) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bfs_cand v = c[i];
    const unsigned g = gap_group(v, g0 ? static_cast<unsigned>(__ldg(g0 + i)) : 0u, maps.m, 3);
    const K w = static_cast<K>(static_cast<unsigned>(v.mwidth) - static_cast<unsigned>(wmin));
    keys[i] = (wbits >= static_cast<int>(8 * sizeof(K)) ? K(0) : static_cast<K>(g) << wbits) | w;
    vals[i] = i;
}

template <typename K>
__global__ void k_gap_offsets(const K* __restrict__ keys, unsigned n, int wbits, unsigned ng, int* __restrict__ offsets) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    auto group = [&](unsigned k) {
        return wbits >= static_cast<int>(8 * sizeof(K)) ? 0u : static_cast<unsigned>(keys[k] >> wbits);
    };
    const unsigned g = group(i);
    if (i == 0 || group(i - 1) != g) offsets[g] = static_cast<int>(i);
    if (i == 0) offsets[ng] = static_cast<int>(n);
}

// Stream-ordered scratch: pieces of one block allocated up front, more blocks
// where it runs out.  What was allocated since a mark can be given back: the
// kernels that used it come before what takes its place on the stream.
struct Scratch {
    cudaStream_t s;
    std::vector<void*> ptrs;
    char* at = nullptr;
    size_t left = 0;
    struct Mark { size_t blocks, left; char* at; };
    Mark mark() const { return {ptrs.size(), left, at}; }
    void release(const Mark& m) {
        for (; ptrs.size() > m.blocks; ptrs.pop_back()) cudaFreeAsync(ptrs.back(), s);
        at = m.at;
        left = m.left;
    }
    bfs_status reserve(size_t bytes) {
        void* p = nullptr;
        bfs_status st = stream_alloc(&p, bytes, s);
        if (st != BFS_OK) return st;
        ptrs.push_back(p);
        at = static_cast<char*>(p);
        left = bytes;
        return BFS_OK;
    }
    bfs_status alloc(void** p, size_t bytes) {
        const size_t need = (bytes + 255) & ~static_cast<size_t>(255);
        if (need > left) {
            char* keep = at;
            const size_t kept = left;
            bfs_status st = reserve(need);
            if (st != BFS_OK) return st;
            *p = at;
            at = keep;
            left = kept;
            return BFS_OK;
        }
        *p = at;
        at += need;
        left -= need;
        return BFS_OK;
    }
    ~Scratch() { for (void* p : ptrs) cudaFreeAsync(p, s); }
};

#define BFS_TRY(x) do { bfs_status st_ = (x); if (st_ != BFS_OK) return st_; } while (0)

}  // namespace
}  // namespace bfs

using namespace bfs;

extern "C" bfs_status bfs_select_delegates(const bfs_cand* d_cands, const int* d_perm, uint32_t n,
                                           const int* d_offsets, uint32_t ngroups,
                                           int* d_delegates, void* stream) {
    BFS_ARG(d_cands && d_perm && d_offsets && d_delegates, "null argument");
    if (ngroups == 0) return BFS_OK;
    BFS_ARG(n > 0 && n < 0x7fffffffu, "bad candidate count %u", n);
    cudaStream_t s = as_stream(stream);
    Scratch sc{s};
    unsigned long long* slots;
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&slots),
                     sizeof(unsigned long long) * kDelegateLanes * ngroups));
    return launch_select_delegates(d_cands, d_perm, n, d_offsets, ngroups, d_delegates, slots, s);
}

static int bits_for(unsigned long long v) {
    int b = 0;
    while (b < 64 && (v >> b) != 0ull) ++b;
    return b;
}

// One pass of the split: sort by (group, field), flag the positions where the
// group changes or the field jumps by more than the metric, and renumber the
// groups.  With sort_only the pass cannot split (the metric is at least the
// field's whole range): the sort alone fixes the member order, the groups and
// their boundaries stay those of the previous pass.
template <typename K>
static bfs_status cluster_pass(const bfs_cand* d_cands, unsigned n, int field, int fmin, int fbits,
                               int end_bit, long long metric, unsigned* gid, bool first, void* kin,
                               void* kout, unsigned* v_in, unsigned* v_out, unsigned* flags,
                               unsigned* scan, void* tmp, size_t tmp_bytes, cudaStream_t s,
                               bool sort_only = false) {
    const int th = 256;
    const int bl = static_cast<int>((n + th - 1) / th);
    K* k_in = static_cast<K*>(kin);
    K* k_out = static_cast<K*>(kout);
    k_pass_keys<K><<<bl, th, 0, s>>>(d_cands, first ? nullptr : gid, n, field, fmin, fbits, k_in, v_in);
    BFS_LAUNCH_CHECK("k_pass_keys");
    size_t b = tmp_bytes;
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(tmp, b, k_in, k_out, v_in, v_out, static_cast<int>(n),
                                             0, end_bit > 0 ? end_bit : 1, s));
    if (sort_only) return BFS_OK;
    k_pass_flags<K><<<bl, th, 0, s>>>(k_out, n, fbits, metric, flags);
    BFS_LAUNCH_CHECK("k_pass_flags");
    b = tmp_bytes;
    BFS_CUDA(cub::DeviceScan::InclusiveSum(tmp, b, flags, scan, static_cast<int>(n), s));
    k_pass_scatter<<<bl, th, 0, s>>>(v_out, scan, n, gid);
    BFS_LAUNCH_CHECK("k_pass_scatter");
    return BFS_OK;
}

// Delegates of the groups (perm / offsets), then sorted by (mt, group).
static bfs_status finish_delegates(const bfs_cand* d_cands, const int* d_perm, unsigned n, const int* d_offsets,
                                   unsigned ng, int tmin, int tbits, int* d_delegates, Scratch& sc, cudaStream_t s) {
    int* dl_group;
    unsigned long long* slots;
    unsigned* u;   // keys, sorted keys, values
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&slots), sizeof(unsigned long long) * kDelegateLanes * ng));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&u), sizeof(unsigned) * 4 * static_cast<size_t>(ng)));
    dl_group = reinterpret_cast<int*>(u + 3 * static_cast<size_t>(ng));
    BFS_TRY(launch_select_delegates(d_cands, d_perm, n, d_offsets, ng, dl_group, slots, s));
    const int th = 256, blg = static_cast<int>((ng + th - 1) / th);
    k_delegate_keys<<<blg, th, 0, s>>>(d_cands, dl_group, ng, tmin, u, u + 2 * static_cast<size_t>(ng));
    BFS_LAUNCH_CHECK("k_delegate_keys");
    size_t b = 0;
    unsigned* dl = reinterpret_cast<unsigned*>(d_delegates);
    // (one start for all: CUB still sorts a bit, and its scratch is asked for with the same bits)
    const int bits = std::max(tbits, 1);
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b, u, u, u, dl, static_cast<int>(ng), 0, bits, s));
    void* tmp;
    BFS_TRY(sc.alloc(&tmp, b));
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(tmp, b, u, u + ng, u + 2 * static_cast<size_t>(ng), dl, static_cast<int>(ng),
                                             0, bits, s));
    return BFS_OK;
}

// The final order by keys of type K: sorts, writes perm and offsets.
template <typename K>
static bfs_status gap_order(const bfs_cand* d_cands, const int* d_group0, unsigned n, const GapMaps& maps, int wmin,
                            int wbits, int end_bit, unsigned ng, int* d_perm, int* d_offsets, Scratch& sc,
                            cudaStream_t s) {
    const int th = 256, bl = static_cast<int>((n + th - 1) / th);
    K* k;
    unsigned* v;
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&k), sizeof(K) * 2 * static_cast<size_t>(n)));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&v), sizeof(unsigned) * static_cast<size_t>(n)));
    k_gap_keys<K><<<bl, th, 0, s>>>(d_cands, d_group0, n, maps, wmin, wbits, k, v);
    BFS_LAUNCH_CHECK("k_gap_keys");
    unsigned* perm = reinterpret_cast<unsigned*>(d_perm);
    size_t b = 0;
    const int bits = end_bit > 0 ? end_bit : 1;
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b, k, k + n, v, perm, static_cast<int>(n), 0, bits, s));
    void* tmp;
    BFS_TRY(sc.alloc(&tmp, b));
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(tmp, b, k, k + n, v, perm, static_cast<int>(n), 0, bits, s));
    k_gap_offsets<K><<<bl, th, 0, s>>>(k + n, n, wbits, ng, d_offsets);
    BFS_LAUNCH_CHECK("k_gap_offsets");
    return BFS_OK;
}

// Groups as the sorting passes form them, from bitmaps of the (group, field)
// cells (*done = false: not applicable).  A pass whose metric is negative
// splits equal values too, and one that needs more than max(2^20, candidates)
// words, or twice that with the passes before, is left to the sorting passes:
// a word takes 8 bytes of scratch until the end and 20 during its pass, so
// the whole stays within the 48 bytes per candidate that those take (the
// final order 32 in place of a pass's 20).  The groups before a pass are
// bounded by the ranges; where that bound asks for more than 2^16 words the
// count is read back (one round trip) instead.
// 0.3 M candidates: two sorting passes 150 us against 45 us.
static bfs_status cluster_by_gaps(const bfs_cand* d_cands, unsigned n, const int* d_group0, unsigned groups0,
                                  const int* metrics, const int* fmin, const long long* range, int* d_perm,
                                  int* d_offsets, int* d_delegates, uint32_t* h_ngroups, Scratch& sc, cudaStream_t s,
                                  bool* done) {
    *done = false;
    for (int f = 0; f < 3; ++f)
        if (metrics[f] < 0) return BFS_OK;
    GapMaps maps{};
    unsigned* total;
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&total), sizeof(unsigned)));
    const int th = 256;
    const unsigned long long most = std::max<unsigned long long>(1ull << 20, n);
    unsigned long long groups = groups0;   // before the pass, at most
    unsigned long long held = 0;           // words of the passes before
    bool exact = true;
    using Count = thrust::counting_iterator<unsigned>;
    using Words = thrust::transform_iterator<GapWord, Count, GapState>;
    for (int f = 0; f < 3; ++f) {
        if (f > 0 && metrics[f] >= range[f]) continue;   // cannot split
        int shift = 5;
        while (shift < 32 && (1ll << shift) <= range[f]) ++shift;
        if (!exact && (groups << (shift - 5)) > (1ull << 16)) {
            unsigned have = 0;
            BFS_TRY(read_back(&have, total, 1, s));
            groups = have;
            exact = true;
        }
        const unsigned long long need = groups << (shift - 5);
        held += need;
        if (shift >= 32 || need > most || held > 2 * most || need > (1ull << 26)) return BFS_OK;
        const unsigned words = static_cast<unsigned>(need);
        const GapRule rule{shift, static_cast<unsigned>(metrics[f])};
        unsigned* bits;
        GapState* state;
        uint2* tab;
        void* tmp;
        size_t tmp_bytes = 0;
        BFS_CUDA(cub::DeviceScan::ExclusiveScan(nullptr, tmp_bytes, Words(Count(0u), GapWord{nullptr, 0u}),
                                                static_cast<GapState*>(nullptr), rule, GapState{0u, 0u, 0u, 0u},
                                                static_cast<int>(words), s));
        BFS_TRY(sc.alloc(reinterpret_cast<void**>(&tab), sizeof(uint2) * static_cast<size_t>(words)));
        // of this pass alone, one piece: states, bits, the scan's own
        const Scratch::Mark pass = sc.mark();
        const size_t at_bits = sizeof(GapState) * static_cast<size_t>(words);
        const size_t at_tmp = (at_bits + sizeof(unsigned) * words + 255) & ~static_cast<size_t>(255);
        char* piece;
        BFS_TRY(sc.alloc(reinterpret_cast<void**>(&piece), at_tmp + tmp_bytes));
        state = reinterpret_cast<GapState*>(piece);
        bits = reinterpret_cast<unsigned*>(piece + at_bits);
        tmp = piece + at_tmp;
        BFS_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned) * words, s));
        const unsigned per_cta = std::max(1024u, ((n + 148 * 4 - 1) / (148 * 4) + 255u) & ~255u);
        k_gap_mark<<<(n + per_cta - 1) / per_cta, 256, 0, s>>>(d_cands, d_group0, n, per_cta, maps, f, fmin[f], shift,
                                                               words, bits);
        BFS_LAUNCH_CHECK("k_gap_mark");
        BFS_CUDA(cub::DeviceScan::ExclusiveScan(tmp, tmp_bytes, Words(Count(0u), GapWord{bits, rule.metric}), state, rule,
                                                GapState{0u, 0u, 0u, 0u}, static_cast<int>(words), s));
        k_gap_table<<<(words + th - 1) / th, th, 0, s>>>(bits, state, words, rule, tab, total);
        BFS_LAUNCH_CHECK("k_gap_table");
        sc.release(pass);
        maps.m[f] = GapMap{tab, fmin[f], shift};
        groups = std::min<unsigned long long>(n, groups * (range[f] / (static_cast<long long>(metrics[f]) + 1) + 1));
        exact = false;
    }
    unsigned ng = 0;
    BFS_TRY(read_back(&ng, total, 1, s));
    BFS_ARG(ng >= 1 && ng <= n, "bad group count %u", ng);
    const int wbits = bits_for(static_cast<unsigned long long>(range[2]));
    const int end_bit = wbits + bits_for(ng - 1);
    const Scratch::Mark order = sc.mark();
    if (end_bit <= 32)
        BFS_TRY(gap_order<unsigned>(d_cands, d_group0, n, maps, fmin[2], wbits, end_bit, ng, d_perm, d_offsets, sc, s));
    else
        BFS_TRY(gap_order<unsigned long long>(d_cands, d_group0, n, maps, fmin[2], wbits, end_bit, ng, d_perm, d_offsets,
                                              sc, s));
    sc.release(order);
    BFS_TRY(finish_delegates(d_cands, d_perm, n, d_offsets, ng, fmin[0],
                             bits_for(static_cast<unsigned long long>(range[0])), d_delegates, sc, s));
    *h_ngroups = ng;
    *done = true;
    return BFS_OK;
}

extern "C" bfs_status bfs_cluster(const bfs_cand* d_cands, uint32_t n, const int* metrics,
                                  int* d_perm, int* d_offsets, int* d_delegates,
                                  uint32_t* h_ngroups, void* stream) {
    return bfs_cluster_grouped(d_cands, n, nullptr, 0, metrics, d_perm, d_offsets, d_delegates,
                               h_ngroups, stream);
}

extern "C" bfs_status bfs_cluster_grouped(const bfs_cand* d_cands, uint32_t n, const int* d_group0,
                                          uint32_t ngroups0, const int* metrics, int* d_perm,
                                          int* d_offsets, int* d_delegates, uint32_t* h_ngroups,
                                          void* stream) {
    BFS_ARG(metrics && h_ngroups, "null argument");
    BFS_ARG(d_group0 == nullptr || ngroups0 >= 1, "ngroups0 must be >= 1 with d_group0");
    *h_ngroups = 0;
    if (n == 0) return BFS_OK;
    BFS_ARG(d_cands && d_perm && d_offsets && d_delegates, "null argument");
    BFS_ARG(n < 0x7fffffffu, "too many candidates");
    cudaStream_t s = as_stream(stream);
    Scratch sc{s};
    // keys, values and the sort's own of the gap grouping, and its small tables
    BFS_TRY(sc.reserve(sizeof(unsigned) * 4 * static_cast<size_t>(n) + (size_t(2) << 20)));
    const int th = 256;
    const int bl = static_cast<int>((n + th - 1) / th);
    // field ranges -> key widths
    int fmin[3];
    long long frange[3];
    unsigned* range;
    unsigned top_group = 0;   // largest initial group
    {
        unsigned h_range[kRanges];
        BFS_TRY(sc.alloc(reinterpret_cast<void**>(&range), sizeof(unsigned) * kRanges));
        BFS_CUDA(cudaMemsetAsync(range, 0, sizeof(unsigned) * kRanges, s));
        const int rb = static_cast<int>((n + kRangeThreads - 1) / kRangeThreads);
        k_field_range<<<std::min(rb, 592), kRangeThreads, 0, s>>>(d_cands, d_group0, n, range);
        BFS_LAUNCH_CHECK("k_field_range");
        BFS_TRY(read_back(h_range, range, kRanges, s));
        top_group = h_range[6];
        for (int f = 0; f < 3; ++f) {
            fmin[f] = static_cast<int>(~h_range[2 * f] ^ 0x80000000u);
            frange[f] = static_cast<long long>(static_cast<int>(h_range[2 * f + 1] ^ 0x80000000u)) - fmin[f];
        }
    }
    bool done = false;
    const Scratch::Mark clean = sc.mark();
    // (the gap tables have cells for groups below ngroups0 only; the sorting passes take any)
    if (!d_group0 || top_group < ngroups0)
        BFS_TRY(cluster_by_gaps(d_cands, n, d_group0, d_group0 ? ngroups0 : 1u, metrics, fmin, frange, d_perm, d_offsets,
                                d_delegates, h_ngroups, sc, s, &done));
    if (done) return BFS_OK;
    sc.release(clean);
    unsigned long long *k_in, *k_out;
    unsigned *v_in, *v_out, *gid, *flags, *scan;
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&k_in), sizeof(unsigned long long) * n));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&k_out), sizeof(unsigned long long) * n));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&v_in), sizeof(unsigned) * n));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&v_out), sizeof(unsigned) * n));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&gid), sizeof(unsigned) * n));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&flags), sizeof(unsigned) * n));
    BFS_TRY(sc.alloc(reinterpret_cast<void**>(&scan), sizeof(unsigned) * n));
    size_t sort64 = 0, sort32 = 0, scan_bytes = 0;
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort64, k_in, k_out, v_in, v_out,
                                             static_cast<int>(n), 0, 64, s));
    BFS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort32, reinterpret_cast<unsigned*>(k_in),
                                             reinterpret_cast<unsigned*>(k_out), v_in, v_out,
                                             static_cast<int>(n), 0, 32, s));
    BFS_CUDA(cub::DeviceScan::InclusiveSum(nullptr, scan_bytes, flags, scan, static_cast<int>(n), s));
    void* tmp;
    const size_t tmp_bytes = std::max(std::max(sort64, sort32), scan_bytes);
    BFS_TRY(sc.alloc(&tmp, tmp_bytes));
    unsigned groups = d_group0 ? ngroups0 : 1u;
    if (d_group0)
        BFS_CUDA(cudaMemcpyAsync(gid, d_group0, sizeof(unsigned) * n, cudaMemcpyDeviceToDevice, s));
    for (int field = 0; field < 3; ++field) {
        const int fbits = bits_for(static_cast<unsigned long long>(frange[field]));
        const int gbits = bits_for(static_cast<unsigned long long>(groups - 1));
        const int end_bit = fbits + gbits;
        // after a pass that numbered the groups, a metric at least the field's
        // whole range (fmax - fmin < 2^fbits) cannot split: sort only
        const bool sort_only = field > 0 && fbits < 62 &&
                               static_cast<long long>(metrics[field]) >= (1LL << fbits);
        bfs_status st;
        if (end_bit <= 32)
            st = cluster_pass<unsigned>(d_cands, n, field, fmin[field], fbits, end_bit,
                                        static_cast<long long>(metrics[field]), gid,
                                        field == 0 && d_group0 == nullptr,
                                        k_in, k_out, v_in, v_out, flags, scan, tmp, tmp_bytes, s, sort_only);
        else
            st = cluster_pass<unsigned long long>(d_cands, n, field, fmin[field], fbits, end_bit,
                                                  static_cast<long long>(metrics[field]), gid,
                                                  field == 0 && d_group0 == nullptr, k_in, k_out,
                                                  v_in, v_out, flags, scan,
                                                  tmp, tmp_bytes, s, sort_only);
        if (st != BFS_OK) return st;
        if (sort_only) continue;   // same groups, same boundaries (groups stay in gid order)
        BFS_TRY(read_back(&groups, scan + (n - 1), 1, s));
    }
    BFS_CUDA(cudaMemcpyAsync(d_perm, v_out, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
    k_offsets<<<bl, th, 0, s>>>(flags, scan, n, d_offsets);
    BFS_LAUNCH_CHECK("k_offsets");
    const unsigned ng = groups;
    BFS_TRY(finish_delegates(d_cands, d_perm, n, d_offsets, ng, fmin[0],
                             bits_for(static_cast<unsigned long long>(frange[0])), d_delegates, sc, s));
    *h_ngroups = ng;
    return BFS_OK;
}
