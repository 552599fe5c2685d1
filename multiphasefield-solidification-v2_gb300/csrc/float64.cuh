// float64.cuh -- float64 conversions and comparisons on the integer pipes.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mpf3d {

// Conversions and comparisons occupy the float64 pipe as long as an addition
// does (16-19 clocks a warp on GB300, measured); the same on the integer
// pipes costs a few issue slots.  Results are those of the conversion and
// comparison instructions.
__device__ __forceinline__ double wide(float x) {
    const uint32_t u = __float_as_uint(x), t = u & 0x7fffffffu;
    if (t - 0x00800000u >= 0x7f000000u)  // zero, subnormal, infinity or NaN
        return t == 0u ? __hiloint2double((int)u, 0) : (double)x;
    return __hiloint2double((int)(((t >> 3) + 0x38000000u) | (u & 0x80000000u)), (int)(u << 29));
}
__device__ __forceinline__ double wide(double x) { return x; }
template <typename T>
__device__ __forceinline__ T narrow(double x);
template <>
__device__ __forceinline__ double narrow<double>(double x) { return x; }
template <>
__device__ __forceinline__ float narrow<float>(double x) {  // round to nearest even
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const uint32_t hi = (uint32_t)(b >> 32), t = hi & 0x7fffffffu;
    if (t - 0x38100000u >= 0x0fd00000u)  // below 2^-126, or near the largest float and beyond
        return (b << 1) == 0u ? __uint_as_float(hi) : (float)x;
    const uint64_t r = (b & 0x7fffffffffffffffull) + 0x0fffffffull + ((b >> 29) & 1u);
    return __uint_as_float((uint32_t)((r >> 29) - 0x1c0000000ull) | (hi & 0x80000000u));
}

__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ float to_float(double x) { return narrow<float>(x); }

constexpr int64_t INF_BITS = 0x7ff0000000000000ll;
// a > b for b >= 0; NaN compares false
__device__ __forceinline__ bool above(double a, double b) {
    const int64_t x = __double_as_longlong(a);
    return x > __double_as_longlong(b) && x <= INF_BITS;
}
// v < 0; NaN compares false
__device__ __forceinline__ bool below_zero(double v) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull;
}
// max(v, 0) with NaN taken to 0, as `if (!(v >= 0)) v = 0`
__device__ __forceinline__ double at_least_zero(double v) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    return b <= (uint64_t)INF_BITS || b == 0x8000000000000000ull ? v : 0.0;
}
// v < floor for v >= 0 (NaN: false)
__device__ __forceinline__ bool below(double v, double floor) {
    return (__double_as_longlong(v) & 0x7fffffffffffffffll) < __double_as_longlong(floor);
}

}  // namespace mpf3d
