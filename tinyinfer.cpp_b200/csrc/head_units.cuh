// A head held as units of four elements: one float4 of its row, or the two halves' elements of two pairs of a turn.
#pragma once

#include "common.cuh"

// Unit u of a head: elements (x0, y0) and (x1, y1) are the pairs of the turn, or four neighbours outside of it.
__device__ __forceinline__ float4 load_unit(const float* p, int u, bool turned, int halves, int half) {
    if (turned && halves) {
        const float2 x = *reinterpret_cast<const float2*>(p + 2 * u), y = *reinterpret_cast<const float2*>(p + 2 * u + half);
        return make_float4(x.x, x.y, y.x, y.y);
    }
    const float4 v = *reinterpret_cast<const float4*>(p + 4 * u);
    return turned ? make_float4(v.x, v.z, v.y, v.w) : v;
}
template <typename T> __device__ __forceinline__ void store2(T* p, float a, float b) {
    if constexpr (sizeof(T) == 2) *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
    else *reinterpret_cast<float2*>(p) = make_float2(a, b);
}
template <typename T>
__device__ __forceinline__ void store_unit(T* p, int u, bool turned, int halves, int half, float4 v) {
    if (turned && halves) {
        store2<T>(p + 2 * u, v.x, v.y);
        store2<T>(p + 2 * u + half, v.z, v.w);
        return;
    }
    if (turned) v = make_float4(v.x, v.z, v.y, v.w);
    store4(p + 4 * u, v);
}
// The unit after the turn by two pairs' (cosine, sine)
__device__ __forceinline__ float4 turn_unit(float4 v, const float2* cs, int u) {
    const float4 f = *reinterpret_cast<const float4*>(cs + 2 * u);
    return make_float4(v.x * f.x - v.z * f.y, v.y * f.z - v.w * f.w, v.z * f.x + v.x * f.y, v.w * f.z + v.y * f.w);
}
