// staged.cuh -- shared-memory plane staging helpers of the stencil kernels:
// zero-filling cp.async copies, the coefficient record types of the level
// precisions, and wrapped coordinates.
#pragma once
#include "common.cuh"

namespace mhdproj {
namespace staged {

// cp.async with zero fill: `valid` false copies nothing and writes zeros,
// which is the value of a cell outside a closed boundary.
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Coefficient records: FP32 float4 (beta_x, beta_y, beta_z, reaction) or four
// FP16/BF16 values packed in 8 bytes.
template <int CK> struct CoefStore { using T = uint2; };
template <> struct CoefStore<0> { using T = float4; };

template <int CK> __device__ __forceinline__ float4 unpack(const typename CoefStore<CK>::T& v);
template <> __device__ __forceinline__ float4 unpack<0>(const float4& v) { return v; }
template <> __device__ __forceinline__ float4 unpack<1>(const uint2& u) {
    const __half2 a = *reinterpret_cast<const __half2*>(&u.x), b = *reinterpret_cast<const __half2*>(&u.y);
    const float2 fa = __half22float2(a), fb = __half22float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
}
template <> __device__ __forceinline__ float4 unpack<2>(const uint2& u) {
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
    const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
}

// Wrapped or absent coordinate along one axis, any number of periods away (a
// halo or the rest of a tile can be wider than the grid).
__host__ __device__ constexpr int axis_wrap(int c, int n, bool periodic, bool* ok) {
    *ok = periodic || (c >= 0 && c < n);
    if (c < 0) return periodic ? n - 1 - (-1 - c) % n : 0;
    if (c >= n) return periodic ? c % n : n - 1;
    return c;
}
// Every coordinate that a tile of 64 columns or 32 rows with its halo reaches
// lands inside the grid, on a periodic axis a whole number of periods away.
constexpr bool axis_wrap_in_range() {
    for (int n = 1; n <= 72; n++)
        for (int c = -8; c < n + 72; c++)
            for (int periodic = 0; periodic < 2; periodic++) {
                bool ok = false;
                const int w = axis_wrap(c, n, periodic != 0, &ok);
                if (w < 0 || w >= n || ok != (periodic || (c >= 0 && c < n)) || (ok && (c - w) % n != 0)) return false;
            }
    return true;
}
static_assert(axis_wrap_in_range(), "a wrapped coordinate leaves the grid");

}  // namespace staged
}  // namespace mhdproj
