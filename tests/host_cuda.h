// The CUDA built-ins that the headers in csrc use, for building them with a host compiler: one
// thread, so that barriers are empty and atomics plain.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#undef __launch_bounds__
#define __launch_bounds__(...)

template <class T, class S>
static inline T bits_as(S s) {
    static_assert(sizeof(T) == sizeof(S), "same size");
    T t;
    std::memcpy(&t, &s, sizeof t);
    return t;
}
static inline int __double2hiint(double x) { return (int)(bits_as<uint64_t>(x) >> 32); }
static inline int __double2loint(double x) { return (int)(uint32_t)bits_as<uint64_t>(x); }
static inline double __hiloint2double(int h, int l) { return bits_as<double>(((uint64_t)(uint32_t)h << 32) | (uint32_t)l); }
static inline double __longlong_as_double(long long v) { return bits_as<double>(v); }
static inline long long __double_as_longlong(double v) { return bits_as<long long>(v); }
static inline float __int_as_float(int v) { return bits_as<float>(v); }
static inline int __float_as_int(float v) { return bits_as<int>(v); }
static inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
static inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
// (a product and a sum kept apart: built with -ffp-contract=off)
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline long long __double2ll_rn(double v) { return std::llrint(v); }
static inline float rsqrtf(float v) { return 1.0f / std::sqrt(v); }
#define __logf(v) std::log(v)
#define __sincosf(v, s, c) (*(s) = std::sin(v), *(c) = std::cos(v))
template <class T> static inline T __shfl_xor_sync(unsigned, T v, int) { return v; }
static inline unsigned atomicMax(unsigned *p, unsigned v) { const unsigned o = *p; *p = std::max(o, v); return o; }
static inline void __syncthreads() {}
using std::isfinite;
static const dim3 threadIdx(0, 0, 0), blockDim(1, 1, 1), blockIdx(0, 0, 0);
