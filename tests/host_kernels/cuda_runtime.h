// Host stand-in for the CUDA runtime header: lets g++ compile a kernel's own
// source so that a test can walk its addresses on the CPU, one thread after
// another.  Inline assembly does nothing (no shared-memory copy happens, so
// the values are meaningless); plain loads and stores are made as written.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <utility>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __grid_constant__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))

struct float2 { float x, y; };
struct alignas(16) float4 { float x, y, z, w; };
struct alignas(16) double2 { double x, y; };
struct uint3 { unsigned x, y, z; };
inline float2 make_float2(float x, float y) { return {x, y}; }
inline double2 make_double2(double x, double y) { return {x, y}; }
inline uint3 threadIdx, blockIdx, blockDim, gridDim;

using std::fma;
using std::max;
using std::min;
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
template <typename T> inline T __ldg(const T* p) { return *p; }
template <typename T> inline T __ldcg(const T* p) { return *p; }
inline double __shfl_down_sync(unsigned, double v, int) { return v; }
inline void __syncthreads() {}
inline void __threadfence() {}
inline unsigned atomicAdd(unsigned* p, unsigned v) { return (*p += v) - v; }
inline int atomicExch(int* p, int v) { return std::exchange(*p, v); }
inline size_t __cvta_generic_to_shared(const void*) { return 0; }

typedef int CUtensorMap;

// asm(...) and asm volatile(...) (keep last: the names are keywords)
#define asm(...) ((void)0)
#define volatile(...) ("")
