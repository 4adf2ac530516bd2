// Internal helpers shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <string>
#include <vector>

#include "bfs.h"

namespace bfs {

// Thread-local last-error message (bfs_last_error()).
void set_error(const char* fmt, ...);
bfs_status fail(bfs_status st, const char* fmt, ...);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// cudaMallocAsync from the device's default pool, which keeps freed memory.
bfs_status stream_alloc(void** p, size_t bytes, cudaStream_t s);

// A few words of pinned host memory of the calling thread, for counts read
// back from the device (kReadBackWords of them; null when pinning failed: the
// caller then reads into pageable memory).
constexpr int kReadBackWords = 16;
unsigned* read_back_words();

// n words from device memory, waiting for the stream.
bfs_status read_back(unsigned* host, const unsigned* d, int n, cudaStream_t s);

#define BFS_CUDA(call)                                                                     \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess)                                                             \
            return ::bfs::fail(BFS_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call,     \
                               cudaGetErrorString(e_));                                    \
    } while (0)

#define BFS_LAUNCH_CHECK(what)                                                             \
    do {                                                                                   \
        cudaError_t e_ = cudaGetLastError();                                               \
        if (e_ != cudaSuccess)                                                             \
            return ::bfs::fail(BFS_ERR_CUDA, "launch of %s failed: %s", what,              \
                               cudaGetErrorString(e_));                                    \
    } while (0)

#define BFS_ARG(cond, ...)                                                                 \
    do {                                                                                   \
        if (!(cond)) return ::bfs::fail(BFS_ERR_ARG, __VA_ARGS__);                         \
    } while (0)

// ---------------------------------------------------------------------------
// FDMT plan (host side).  Built once per (fmin, fmax, nchan, ncols, max_dt).
// ---------------------------------------------------------------------------
struct FdmtLevel {
    int nsub = 0;                 // sub-bands at this level
    std::vector<int> rows;        // rows per sub-band
    std::vector<int> cum;         // nsub + 1 cumulative rows
    std::vector<float> freq;      // nsub + 1 sub-band edges (MHz)
    // level >= 1: one entry per output row (global indices in the previous plane)
    std::vector<int> a_row, b_row, shift;
    // maximum look-back (samples) of any row of this level, counting level 0
    std::vector<int> lookback;    // per row
    int total_rows() const { return cum.empty() ? 0 : cum[nsub]; }
};

struct FdmtPlanHost {
    int kind = BFS_PLAN_KEITH;
    float fmin = 0, fmax = 0;
    int nchan = 0, ncols = 0, max_dt = 0;
    int niter = 0;
    int rows_per_chan0 = 0;  // level-0 rows of every channel (d0 + 1); Pravir plans: 0
                             // (per channel: lv[0].rows, delays dt0)
    std::vector<int> dt0;    // Pravir plans: the delay of every level-0 row
    std::vector<int> dt_out; // delay of every output row
    std::vector<FdmtLevel> lv;  // niter + 1 levels
    int out_rows() const { return lv.empty() ? 0 : lv.back().total_rows(); }
};

// Builds the plan exactly as the reference's CFdmtB/CFdmtCpu do.  Returns
// BFS_OK or BFS_ERR_ARG (with the message set).
bfs_status build_fdmt_plan(float fmin, float fmax, int nchan, int ncols, int max_dt,
                           FdmtPlanHost* out);
// The reference's second FDMT variant (FDMT_PRAVIR): delay grids dt_min ..
// dt_max step dt_step per sub-band, window-mean level 0, rounded mid-band
// mappings.  BFS_ERR_ARG where the reference throws.
bfs_status build_pravir_plan(float fmin, float fmax, int nchan, int ncols, int dt_max, int dt_step,
                             int dt_min, FdmtPlanHost* out);

// Inverse row tables of the adjoint: for level l >= 1 and every row i of the
// level-(l-1) plane, the level-l rows g that read row i, with the shift of
// the read (0 as the tail row a_g, s_g as the head row b_g), in ascending g.
struct AdjointTables {
    std::vector<size_t> off_pos;  // per level: start of its nrows+1 offsets in `off`
    std::vector<size_t> ent_pos;  // per level: start of its entries in `ent`
    std::vector<int> off;         // CSR offsets (relative to the level's entries)
    std::vector<int> ent;         // pairs {g, shift}
    bool built = false;
};
void build_adjoint_tables(const FdmtPlanHost& p, AdjointTables* out);

// ---------------------------------------------------------------------------
// Adjoint run segment: the gradient of level l1 taken down to level l0 in one
// pass over HBM, as two stages of one or two levels (S1 = l1 -> mid, S2 = mid
// -> l0).  A row of a stage is a sum of shifted rows above it, nested as the
// levels are: for two levels sum over the rows g that read it of (sum over
// the rows h that read g of h[u + s_h]), each sum from +0 in ascending row
// order; terms past ncols are zeros (x + 0 is x for every partial sum, none
// of which is -0).  With `final` the outputs are channels: the level-0 rows'
// running-mean adjoint is folded in, row r' of a channel being summed again
// at each of its r' + 1 offsets.
//
// A level-l1 row is read at shift 0 by a tail row and at up to the whole
// sub-band's delay by a head row, so a tile's output row i has a window of
// its own, samples t0 - E_i .. t0 - E_i + kSegTile - 1 with E_i the least
// total shift of its terms (a multiple of 8 below it): all windows of the
// tile then read the level-l1 rows at [t0, t0 + kSegTile + a few).  Time tiles
// run until t0 - E_i passes the row's end.  A tile holds the outputs whose
// first reader lies in a cut of consecutive level-l1 rows (channels stay
// whole).  X holds the level-l1 rows, pitch_x floats each, the row's window
// starting `lead` samples before t0; Y the mid rows, kRunMid floats each.
//
// blob (ints, per tile, staged in shared memory): per mid row the index of its
// terms | its kind, then {row, E, index | kind} per output, then the terms,
// every row's from a multiple of 4: byte offset | 1 (last of an inner sum) |
// 2 (final: last term of a level-0 row's value) | r' << 20 | r << 23 | 1 << 26
// (last of row r') | kAdjEnd (last of the row).
// ---------------------------------------------------------------------------
enum { kAdjTerms = 0, kAdjPairs = 1, kAdjOnes = 2, kAdjZero = 3 };  // two sums of two / of one term; no term
constexpr int kAdjEnd = 1 << 28;

struct AdjTile {                 // device-side
    int row;                     // first of its input rows
    int blob;                    // first int of its blob (a multiple of 4)
    int len;                     // ints of it, a multiple of 4
    int n_in, n1, n2;
    int max_e;                   // largest E
    int pad;
};

struct AdjRun {
    int l0 = 0, l1 = 0;
    bool final = false;
    int pitch_x = 0, y0 = 0, blob0 = 0, max_blob = 0, max_e = 0;
    size_t smem_bytes = 0;
    std::vector<AdjTile> tiles;
    std::vector<int> rows;       // 2 ints per input row: {plane row, lead}
    std::vector<int> blob;
};
// rows: outputs per tile, tried in order until one fits; in_pitch: floats per
// level-l1 row (the caller's plane: ncols), which fixes the leads.
bool build_adj_run(const FdmtPlanHost& p, const AdjointTables& t, int l0, int l1, bool final,
                   const std::vector<int>& rows, int in_pitch, size_t smem_limit, AdjRun* out);

// FDMT of 0/1 rows: every level-0 value of a 0/1 row is exactly 0 or 1 and
// every merge adds integers, so output row d at sample t is exactly the
// number of channels c with weight 1 whose total delay along the merge tree,
// tau(d, c) (the level-0 row plus every head shift on the path), is <= t.
// tau is row-major [out_row][channel]; max_tau its largest value.
void build_ones_delays(const FdmtPlanHost& p, std::vector<int>* tau, int* max_tau);

// ---------------------------------------------------------------------------
// Fused "head" of the FDMT: levels 0..k of one group of 2^k adjacent channels
// computed by one CTA over a time tile, all intermediate levels in shared
// memory.  Tables index rows local to the group's shared-memory planes.
// ---------------------------------------------------------------------------
constexpr int kHeadMaxDepth = 8;

struct HeadGroup {                  // device-side, one per channel group
    int halo;                       // samples of look-back of the group's level-k rows
    int out_row0;                   // first row of the group's sub-band in the level-k plane
    int rows[kHeadMaxDepth + 1];    // rows of the group at levels 0..k
    int tab_off[kHeadMaxDepth + 1]; // offset of level l's table (l >= 1)
};

struct HeadPlan {
    int depth = 0;          // k (0 = no fused head)
    int group = 1;          // 2^k channels per CTA
    int tile = 0;           // output samples per CTA
    int width = 0;          // tile + max halo, rounded to a warp: threads per CTA
    int rows_a = 0;         // shared rows of the even-level buffer (level 0, 2, ...)
    int rows_b = 0;         // shared rows of the odd-level buffer (>= group: it first
                            // stages the group's input rows)
    int tab_rows = 0;       // largest per-group table (levels 1..k), staged in shared memory
    size_t smem_bytes = 0;
    std::vector<HeadGroup> groups;
    std::vector<int> tab;   // 4 ints per row: {a_local, b_local, shift, 0}
};

// Head plan for depth k and tile width; returns false when k is not usable
// (k > trailing zero bits of nchan, k > niter, or too much shared memory).
bool build_head_plan(const FdmtPlanHost& p, int k, int tile, size_t smem_limit, HeadPlan* out);

// ---------------------------------------------------------------------------
// Fused merge segment: levels l0+1..l1 in one pass over HBM.  The level-l1
// plane is cut into tiles of `rows` consecutive rows x `tile` samples.  For
// one such tile the rows of levels l0..l1-1 it depends on (a row DAG through
// the merge tables) are held in shared memory, each over its own window of
// samples: a row reached from the tile's rows through head shifts between
// lo and hi samples in total needs the samples [t0 - hi, t0 + tile - lo),
// which is `tile` + (hi - lo) columns wide, and hi - lo stays small (the
// shifts of neighbouring rows differ by a sample or two), however large the
// shifts themselves are.  So any adjacent levels fuse, the last ones
// included, with only the level-l0 rows read from HBM and the level-l1
// rows written.
// ---------------------------------------------------------------------------
constexpr int kSegMaxLevels = 6;
constexpr int kSegTile = 256;    // output samples per segment tile
constexpr int kSegMaxChunks = 12;  // 32-column chunks per shared row at most

struct SegTile {                 // device-side, one per row tile of a segment
    int ent;                     // first entry of the tile in the segment's entries
    int n[kSegMaxLevels + 1];    // n[0] input rows, n[i] rows of level l0 + i (n[m]: output)
};

// Shared memory: three buffers X0, Y, X1, each of its rows, then a row of
// -0.0 (x + -0 == x bit for bit: the head row of rows without one) and a
// guard row (a chunk of the last row may read up to one pitch past it, in
// columns no written sample depends on); then the entries of two tiles.
// Level i of a tile is held in X (i even) or Y (i odd); a CTA runs tiles one
// after another, loading the next tile's input rows into the other X buffer
// while it merges the current one.  Entries, 4 ints each, in the tile's
// order: n[0] input rows {plane row, window lead E (a multiple of 4, so each
// row's window starts on a 16-byte boundary of the plane), 0, offset in X},
// then for every level i = 1..m its rows {offset of the tail row's sample and
// of the head row's sample minus the shift, both in the buffer of level
// i-1, first sample that adds the head row relative to t0 (shift + lead),
// destination: offset in the buffer of level i, or the plane row at level
// m}.  Offsets count floats; local column u of a row with lead E holds
// sample t0 - E + u.
struct SegPlan {
    int l0 = 0, l1 = 0;
    int rows = 0;                // output rows per tile
    int tile = 0;                // output samples per tile (multiple of 32)
    int nc = 0;                  // 32-column chunks per shared row
    int pitch = 0;               // floats per shared row (32 nc)
    int rows_x = 0, rows_y = 0;  // rows of buffer X (levels l0, l0+2, ..) and Y (l0+1, ..)
    int size_x = 0, size_y = 0;  // floats of a buffer: its rows, the -0.0 row, the guard row
    int max_thr = 0;             // tiles with t0 >= max_thr never need the t >= shift test
    int threads = 0;             // CTA size of its kernel (0: 256 when two CTAs fit an SM, else 512)
    bool single = false;         // one input buffer: the next tile loads after this one is merged
    int r0c = 0;                 // input segment (levels 1..l1 straight from the channels):
                                 // level-0 rows per channel; 0 = the input is a level plane
    int max_in_rows = 0;         // most input rows of one tile
    int64_t in_rows = 0;         // input rows summed over tiles (HBM reads per time tile)
    int y0 = 0, x1 = 0;          // offsets of buffers Y and X1 (X0 is at 0)
    int ent_base = 0;            // offset (floats) of the two staged entry buffers
    int max_ent = 0;             // most entries of one tile
    size_t smem_bytes = 0;
    std::vector<SegTile> tiles;
    std::vector<int> ent;
};

// Input segment (from_input, BFS_PLAN_KEITH, l0 = 0): the tile's input rows
// are channels of the filterbank, each over the window its level-0 rows need
// (r more samples on the left for the running mean of row r), and level 1
// is formed straight from them: a level-1 entry's w packs the destination
// (low 20 bits), the tail and head rows' level-0 row numbers (4 bits each at
// 20 and 24) and the shift (4 bits at 28); its x / y point at sample t of the
// tail channel and t - shift of the head channel.  No level-0 plane exists.
//
// Segment plan for levels l0+1..l1 with `rows` output rows and `tile`
// samples per tile; false when it needs more than kSegMaxLevels levels,
// kSegMaxChunks chunks per row or smem_limit bytes of shared memory (or, for
// an input segment, a level-0 depth, shift or offset beyond its packing).
bool build_seg_plan(const FdmtPlanHost& p, int l0, int l1, int rows, int tile, size_t smem_limit,
                    SegPlan* out, bool from_input = false, bool single = false);

// ---------------------------------------------------------------------------
// Run segment: levels l0+1..l1 (two, three or four) in one pass over HBM, as
// two stages of one or two merge levels each.  A stage forms a row from the
// two or four rows below it at once, in registers: with two levels,
//   out[t] = (A[t] + B[t - p]) + (C[t - q] + D[t - q - r])
// (the adds of the two levels, each rounded as there).  Consecutive rows of
// a sub-band step along a staircase through the tables: from one row to the
// next either the tail changes or the head does, so most of the four inputs
// stay where they were and are kept in registers; an entry says which of
// them moved.  Stage 1 goes from the input rows (buffer X) to the mid level
// (buffer Y), stage 2 from there to HBM.
//
// A tile is `n2` consecutive rows of the level-l1 plane from row out0 on (cut
// at sub-band borders, so its mid rows belong to few sub-bands) x kSegTile
// samples.  The mid rows of one sub-band share one window (samples
// t0 - hi .. ), which keeps an unchanged input at one offset from row to row.
// X holds the input rows, `pitch_x` floats each, then a row of -0.0 (the head
// of rows without one); samples before 0 hold -0.0 as well, so no merge
// tests t >= shift: x + -0 is x bit for bit.  Y holds the mid rows, kRunMid
// floats each, then its -0.0 row.  Each buffer's -0.0 row is long enough for
// a read of its last row that runs past the row's end (columns no written
// sample depends on).
// Input segments (r0c > 0; Keith plans, and Pravir plans with delays 0, 1,
// 2, .. per channel): the input rows are channels and an input of stage 1 is
// a level-0 row of one: entry bits 20.. give its row number r, the
// running mean over r + 1 samples is formed where it is read.
// 16-bit plans (esize 2) keep both buffers in 16 bits: offsets and pitches
// count 2-byte values, tiles have kRun16Tile samples and mid rows kRun16Mid,
// windows start on 16-byte boundaries (8 samples).
// ---------------------------------------------------------------------------
constexpr int kRunMidChunks = 9;                  // 32-column chunks of a mid row
constexpr int kRunMid = 32 * kRunMidChunks;
constexpr int kRunOutChunks = kSegTile / 32;
constexpr int kRunMaxPitch = 384;
constexpr int kRun16Tile = 2 * kSegTile;          // 16-bit plans: the same bytes per row
constexpr int kRun16Mid = 2 * kRunMid;
constexpr int kRun16Over = 72;                    // values past its last input row that a tile may read (cleared)

struct RunTile {                 // device-side
    int row;                     // first of the tile's input rows
    int ent;                     // first of its entries: n1 of stage 1, then n2 of stage 2
    int n_in, n1, n2;
    int out0;                    // first row in the level-l1 plane
    int pad[2];
};

struct RunPlan {
    int l0 = 0, l1 = 0;
    int s1 = 0, s2 = 0;          // levels merged by each stage (0: no plan)
    int esize = 4;               // bytes of a value in the planes and buffers
    int r0c = 0;                 // input segment: most level-0 rows of a channel
    bool positive = false;       // input segment of a Pravir plan: its window sums start at +0,
                                 // so a channel's -0.0 counts as +0
    int pitch_x = 0;             // values per row of X
    int zero_x = 0, zero_y = 0;  // offsets of the -0.0 rows
    int y0 = 0, ent0 = 0;        // offsets of Y and of the two staged entry buffers
    int max_ent = 0;             // most entries of one tile
    int edge = 0;                // tiles with t0 >= edge read no sample before the last level-0 row number
    size_t smem_bytes = 0;
    std::vector<RunTile> tiles;
    std::vector<int> rows;       // 2 ints per input row: {plane row, lead}: its window starts at t0 - lead
    std::vector<int> ent;        // 4 ints per entry: byte offsets of the inputs | 1 where it moved | r << 20
};

// False when a window, a row or smem_limit does not allow it.  ncols fixes
// the leads of an input segment: a channel's window starts on a 16-byte
// boundary of the filterbank, whose rows are ncols floats.
bool build_run_plan(const FdmtPlanHost& p, int l0, int l1, int rows, size_t smem_limit, RunPlan* out,
                    bool from_input, int esize = 4);

// bfs_preproc_calc_fdmt_inputs with the mask as one value (0 or 1) per row.
bfs_status clean_rows(float* x, int nrows, int ncols, float* buff, float* row_mask, cudaStream_t s);
// Whether the plan's row-mask FDMT can run (its delay table built on first
// use), and out /= sqrt(row-mask FDMT + 1e-8) in place, as
// bfs_fdmt_execute_row_mask and bfs_fdmt_normalize form it.
bfs_status row_mask_ready(bfs_fdmt_plan* plan);
bfs_status row_mask_normalize(bfs_fdmt_plan* plan, const float* row_mask, float* out, cudaStream_t s);

}  // namespace bfs
