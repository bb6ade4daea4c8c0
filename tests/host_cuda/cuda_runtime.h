// Host stand-ins for the few CUDA device functions that fastmath.cuh and
// smallstep.cuh use, so that their arithmetic can be checked on the CPU
// (tests/test_smallstep_host.py; compiled with -ffp-contract=off).  The special-
// function unit's reciprocal square root is a correctly rounded one off by up
// to one unit in the last place, by turns.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline
#define __noinline__

template <typename T, typename U>
inline T bits_as(U u)
{
    T t;
    static_assert(sizeof(T) == sizeof(U), "sizes");
    std::memcpy(&t, &u, sizeof t);
    return t;
}

inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float __frcp_rn(float x) { return 1.0f / x; }
inline int __double2hiint(double d) { return (int)(bits_as<int64_t>(d) >> 32); }
inline int __double2loint(double d) { return (int)bits_as<int64_t>(d); }
inline double __hiloint2double(int h, int l) { return bits_as<double>((int64_t)(((uint64_t)(uint32_t)h << 32) | (uint32_t)l)); }
inline float __int_as_float(int i) { return bits_as<float>(i); }
inline float __uint_as_float(unsigned i) { return bits_as<float>(i); }
inline int __float_as_int(float f) { return bits_as<int>(f); }
inline unsigned __float_as_uint(float f) { return bits_as<unsigned>(f); }
inline long long __double_as_longlong(double d) { return bits_as<long long>(d); }
inline double __longlong_as_double(long long d) { return bits_as<double>(d); }
inline int __clz(unsigned x) { return x ? __builtin_clz(x) : 32; }
inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s)
{
    return (unsigned)((((uint64_t)hi << 32 | lo) << s) >> 32);
}
inline float rsqrtf(float x)
{
    static int turn = 0;
    turn = (turn + 1) % 3;
    return bits_as<float>(bits_as<int>((float)(1.0 / std::sqrt((double)x))) + turn - 1);
}
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
template <typename T>
inline T min(T a, T b) { return a < b ? a : b; }
