// Launch of a run segment (fdmt_run.cu) for the FDMT's schedules.
#pragma once
#include <cuda_runtime.h>

#include "internal.h"

namespace bfs {

// One pass of rp over ncols samples: src (the level-l0 plane, or the
// filterbank of an input segment; ones: not read, the all-ones image) to dst.
// Planes other than the caller's have a pitch of whole 128-byte lines.
cudaError_t launch_run(const RunPlan& rp, const float* src, float* dst, const RunTile* tiles, const int2* rows,
                       const int4* ent, int ncols, int in_pitch, int out_pitch, int ones, cudaStream_t s);

// The same over 16-bit planes of a plan whose level-l rows all carry the scale
// 2^-l: src and, unless out_f32, dst hold S = __half or __nv_bfloat16.
template <typename S>
cudaError_t launch_run16(const RunPlan& rp, const S* src, void* dst, bool out_f32, const RunTile* tiles,
                         const int2* rows, const int4* ent, int ncols, int in_pitch, int out_pitch, cudaStream_t s);

}  // namespace bfs
