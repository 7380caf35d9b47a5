// The CUDA functions that the traversal headers use, for the host compiler: every rounding as on the
// device (plain float operations with -ffp-contract=off, std::fma, and an exact round-down add).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __global__
#define __forceinline__ inline
#define __restrict__
#define __align__(n) alignas(n)
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
inline float2 make_float2(float a, float b) { return {a, b}; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __frcp_rn(float a) { return 1.0f / a; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __fdividef(float a, float b) { return a / b; }
inline float __fadd_rd(float a, float b) {  // the double sum of two floats of these ranges is exact
    const double s = (double)a + (double)b;
    float r = (float)s;
    return (double)r > s ? std::nextafterf(r, -INFINITY) : r;
}
inline float2 __fadd2_rn(float2 a, float2 b) { return {a.x + b.x, a.y + b.y}; }
inline float2 __fmul2_rn(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)}; }
inline float2 __fadd2_rd(float2 a, float2 b) { return {__fadd_rd(a.x, b.x), __fadd_rd(a.y, b.y)}; }
inline int __float_as_int(float f) { int i; std::memcpy(&i, &f, 4); return i; }
inline int __float2int_rd(float f) { return (int)std::floor(f); }
inline float __expf(float x) { return std::exp(x); }
inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
using std::isfinite;
using std::max;
using std::min;
struct { int x; } static threadIdx;
inline float __shfl_xor_sync(unsigned, float v, int, int) { return v; }
inline float __ldg(const float *p) { return *p; }
inline void atomicAdd(float *p, float v) { *p += v; }
typedef void *cudaStream_t;
