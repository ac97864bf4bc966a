// Device helpers of the table path's edge kernels.
#pragma once
#include <type_traits>
#include "tab.cuh"
#include "tc_layout.cuh"

namespace mlff {

// dt/dd of the table's local coordinate, as the kernels use it in FP32; the
// build places its nodes with the same rounded value.
__host__ __device__ inline float tab_scale(float cutoff) { return (float)(2.0 * TAB_NI / (double)cutoff); }

// Two FP32 values in a register pair and their two-wide fused multiply-add:
// one instruction slot for two roundings-to-nearest fused multiply-adds.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(f32x2 v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo;
}
__device__ __forceinline__ float hi2(f32x2 v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return hi;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// A condition that is the same in every lane, as a vote: the branch on it
// needs no divergence bookkeeping and is not turned into predicated code.
__device__ __forceinline__ bool uni(bool p) { return __any_sync(0xffffffffu, p); }

// f(integral_constant<int, r>) for a warp-uniform r < G, so that
// per-receiver sums stay in registers
template <int G, int BASE = 0, class F>
__device__ __forceinline__ void tab_switch(int r, F&& f) {
    if constexpr (G == 1) {
        f(std::integral_constant<int, BASE>{});
    } else {
        if (uni((r & (G / 2)) != 0)) tab_switch<G / 2, BASE + G / 2>(r, f);
        else tab_switch<G / 2, BASE>(r, f);
    }
}

// Sums of 16 per-lane values over the warp's lanes with 16 shuffles
// (reduce-scatter): lanes 2 i and 2 i + 1 return the sum of v[i].
__device__ __forceinline__ float reduce16(const float (&v)[16], int lane) {
    float a[8], b[4], c[2];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4, h2 = lane & 2;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        a[j] = (h16 ? v[j + 8] : v[j]) + __shfl_xor_sync(0xffffffffu, h16 ? v[j] : v[j + 8], 16);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        b[j] = (h8 ? a[j + 4] : a[j]) + __shfl_xor_sync(0xffffffffu, h8 ? a[j] : a[j + 4], 8);
#pragma unroll
    for (int j = 0; j < 2; ++j)
        c[j] = (h4 ? b[j + 2] : b[j]) + __shfl_xor_sync(0xffffffffu, h4 ? b[j] : b[j + 2], 4);
    float s = (h2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h2 ? c[0] : c[1], 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

}  // namespace mlff
