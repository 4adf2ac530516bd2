// Rows of 32-column chunks in registers and shared memory: lane l of a warp
// holds columns l, l + 32, .. (every shared access is one wavefront whatever
// the row's offset).  Used by the run segments of the FDMT and its adjoint.
#pragma once

#include <cuda_runtime.h>

namespace bfs {

__device__ __forceinline__ void copy16(unsigned s, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy4(unsigned s, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Both halves rounded to nearest, each exactly as __fadd_rn.
__device__ __forceinline__ void add2(float& o0, float& o1, float a0, float a1, float b0, float b1) {
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(o0), "=f"(o1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

template <int K>
__device__ __forceinline__ void add_rows(float (&o)[K], const float (&a)[K], const float (&b)[K]) {
#pragma unroll
    for (int k = 0; k + 1 < K; k += 2) add2(o[k], o[k + 1], a[k], a[k + 1], b[k], b[k + 1]);
    if constexpr (K % 2 == 1) o[K - 1] = __fadd_rn(a[K - 1], b[K - 1]);
}

template <int K>
__device__ __forceinline__ void load_row(float (&v)[K], const char* p) {
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = *reinterpret_cast<const float*>(p + 128 * k);
}

}  // namespace bfs
