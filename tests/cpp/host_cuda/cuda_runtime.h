// The part of CUDA's language that the kernels' per-point functions use, as plain C++: a
// CPU test then runs those functions themselves, with a sanitizer on the memory they read.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#define __host__
#define __device__
#define __global__
#define __shared__
#define __restrict__
#define __forceinline__ inline
#define __noinline__
#define __align__(n) __attribute__((aligned(n)))
#define __launch_bounds__(...)

struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct alignas(16) double2 { double x, y; };
struct uint4 { unsigned x, y, z, w; };
struct dim3 { unsigned x, y, z; };
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline double2 make_double2(double x, double y) { return {x, y}; }
inline dim3 threadIdx, blockIdx, blockDim, gridDim;

inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline float __fdividef(float a, float b) { return a / b; }
inline float __logf(float x) { return std::log(x); }
inline void __sincosf(float x, float* s, float* c) { *s = std::sin(x); *c = std::cos(x); }
inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
template <class T> T __ldg(const T* p) { return *p; }
template <class T> T atomicCAS(T* p, int old, int v) { const T o = *p; if (o == (T)old) *p = (T)v; return o; }
template <class T> T atomicAdd(T* p, unsigned v) { const T o = *p; *p += v; return o; }
template <class T> T atomicExch(T* p, int v) { const T o = *p; *p = (T)v; return o; }
inline void __syncthreads() {}
inline void __threadfence() {}
inline void __nanosleep(unsigned) {}
template <class T> size_t __cvta_generic_to_shared(const T* p) { return (size_t)p; }
