// What the two tensor-core kernels of the attention with options have in common: the exponential and reciprocal of the
// cap, the first key that a position sees, and the cut of a softmax weight into three bfloat16 parts.
#pragma once

#include "common.cuh"

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// The first key that position p sees, through a window and/or chunks of positions (0: none).
__device__ __forceinline__ int first_key_seen(int p, int window, int chunk) {
    int lo = window > 0 ? max(0, p - window + 1) : 0;
    if (chunk > 0) lo = max(lo, p / chunk * chunk);
    return lo;
}
// Two floats as three pairs of bfloat16 whose sums are the floats: the upper 16 bits of a float
// are a bfloat16 (truncated), what is left is exact in float32 and is cut the same way again;
// after three cuts nothing of the 24-bit significand is left.
__device__ __forceinline__ void split3_pair(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
    const unsigned xb = __float_as_uint(x), yb = __float_as_uint(y);
    hi = __byte_perm(xb, yb, 0x7632);
    const float x1 = x - __uint_as_float(xb & 0xffff0000u), y1 = y - __uint_as_float(yb & 0xffff0000u);
    const unsigned x1b = __float_as_uint(x1), y1b = __float_as_uint(y1);
    mid = __byte_perm(x1b, y1b, 0x7632);
    const float x2 = x1 - __uint_as_float(x1b & 0xffff0000u), y2 = y1 - __uint_as_float(y1b & 0xffff0000u);
    lo = __byte_perm(__float_as_uint(x2), __float_as_uint(y2), 0x7632);
}
