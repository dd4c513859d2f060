"""The CUDA built-ins of the generated modules as host C++, for tests that
compile a module's source (or a part of it) with the host compiler."""

INTRINSICS = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __global__
#define __constant__
#define __shared__
#define __noinline__
#define __forceinline__ inline
#define __launch_bounds__(...)
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
template <class T, class S> static inline T as(S s) { T t; std::memcpy(&t, &s, sizeof t); return t; }
static inline long long __double_as_longlong(double x) { return as<long long>(x); }
static inline double __longlong_as_double(long long x) { return as<double>(x); }
static inline unsigned __float_as_uint(float x) { return as<unsigned>(x); }
static inline float __uint_as_float(unsigned x) { return as<float>(x); }
static inline float gpu_log2f(float x) { return std::log2(x); }
#define __log2f gpu_log2f
static inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
static inline int __popc(unsigned x) { return __builtin_popcount(x); }
"""
