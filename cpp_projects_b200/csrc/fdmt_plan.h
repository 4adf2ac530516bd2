// The FDMT plan object behind the opaque bfs_fdmt_plan handle (shared by the
// forward and adjoint translation units).
#pragma once
#include <cuda_runtime.h>

#include <array>
#include <cstring>
#include <utility>
#include <vector>

#include "internal.h"

namespace bfs {
// Host tables gathered for one device allocation and one copy.
class TableUpload {
public:
    template <typename T> void add(T** dst, const std::vector<T>& v) {
        if (v.empty()) return;
        const size_t at = (bytes_.size() + 255) & ~static_cast<size_t>(255);
        bytes_.resize(at + v.size() * sizeof(T));
        std::memcpy(bytes_.data() + at, v.data(), v.size() * sizeof(T));
        refs_.push_back({reinterpret_cast<void**>(dst), at});
    }
    // *arena owns the memory (cudaFree); the added pointers address it
    bfs_status commit(void** arena) {
        if (bytes_.empty()) return BFS_OK;
        BFS_CUDA(cudaMalloc(arena, bytes_.size()));
        BFS_CUDA(cudaMemcpy(*arena, bytes_.data(), bytes_.size(), cudaMemcpyHostToDevice));
        for (auto& r : refs_) *r.first = static_cast<char*>(*arena) + r.second;
        return BFS_OK;
    }
private:
    std::vector<unsigned char> bytes_;
    std::vector<std::pair<void**, size_t>> refs_;
};
}  // namespace bfs

struct bfs_fdmt_plan {
    bfs::FdmtPlanHost host;
    int device = -1;
    bool host_only = false;
    bool external_ws = false;
    int fuse_depth = 0;
    int precision = BFS_PREC_F32;      // storage of the planes between levels
    void* d_tables = nullptr;          // owns the forward's tables (the pointers below into it)
    int4* d_tab = nullptr;             // per level, per output row: {a, b, shift, exps}
    std::vector<size_t> tab_off;       // offset of each level's table in d_tab
    void* d_buf[2] = {nullptr, nullptr};
    size_t buf_rows[2] = {0, 0};
    size_t ws_bytes = 0;
    bfs::HeadPlan head;                     // fused levels 0..k (depth 0 = not used)
    bfs::HeadGroup* d_head_groups = nullptr;
    int* d_head_tab = nullptr;
    // passes after the head (or level 0): a fused segment of levels l0+1..l1
    // (tiles non-empty) or one plain merge level (l1 = l0 + 1, no tiles)
    std::vector<bfs::SegPlan> passes;
    std::vector<bfs::RunPlan> runs;    // per pass: its run segment (s1 = 0: k_fdmt_seg or a plain level)
    std::vector<int> plane_buf;        // per level: ping-pong plane holding it in HBM (-1: never)
    bfs::SegTile* d_seg_tiles = nullptr;  // every fused segment's tiles, concatenated
    int* d_seg_ent = nullptr;          // every fused segment's entries, concatenated
    std::vector<size_t> seg_tile0, seg_ent0;  // per pass: offsets into the two arrays
    bfs::RunTile* d_run_tiles = nullptr;  // every run segment's tiles, input rows and entries
    int* d_run_rows = nullptr;
    int* d_run_ent = nullptr;
    std::vector<size_t> run_tile0, run_row0, run_ent0;
    int* d_lvl0 = nullptr;             // Pravir plans: level-0 row cumsum (nchan+1) then delays
    int* d_ones_tau = nullptr;         // FDMT of 0/1 rows: tau [out_row][channel] (first use)
    int ones_max_tau = -1;
    // adjoint (built on the first adjoint call): per level l >= 1, for every
    // row of level l-1 the level-l rows that read it, as CSR {row, shift}
    bfs::AdjointTables adj;
    void* d_adj_tables = nullptr;      // owns the adjoint's tables
    int* d_adj_off = nullptr;
    int2* d_adj_ent = nullptr;
    std::vector<bfs::AdjRun> adj_runs;   // run segments from the top level down (empty: a pass per level)
    bfs::AdjTile* d_adj_tiles = nullptr;
    int* d_adj_rows = nullptr;
    int* d_adj_blob = nullptr;
    std::vector<std::array<size_t, 3>> adj_run0;  // per segment: offsets into the three arrays
    void* d_adj_buf[2] = {nullptr, nullptr};  // plan-owned adjoint planes (bfs_fdmt_adjoint)
    ~bfs_fdmt_plan() {
        if (d_tables) cudaFree(d_tables);
        if (d_adj_tables) cudaFree(d_adj_tables);
        if (d_ones_tau) cudaFree(d_ones_tau);
        for (void* b : d_buf)
            if (b) cudaFree(b);
        for (void* b : d_adj_buf)
            if (b) cudaFree(b);
    }
};
