// Stand-ins for the CUDA builtins that the device headers name, so that a host
// compiler can build the parts of them that one thread runs on its own: one
// block of one thread; what only a warp can do is declared, not defined.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef __noinline__
#define __noinline__
#endif

inline float __int_as_float(int v)
{
    float f;
    memcpy(&f, &v, sizeof f);
    return f;
}
inline double __longlong_as_double(long long v)
{
    double d;
    memcpy(&d, &v, sizeof d);
    return d;
}
#include <math_constants.h>

struct HostIdx {
    int x, y, z;
};
static const HostIdx threadIdx{0, 0, 0}, blockIdx{0, 0, 0}, blockDim{1, 1, 1}, gridDim{1, 1, 1};

using std::max;
using std::min;

template <typename T>
inline T __ldg(const T *p)
{
    return *p;
}
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline float __fdividef(float a, float b) { return a / b; }
inline float __frcp_rn(float a) { return 1.0f / a; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }

int __any_sync(unsigned, int);
unsigned __ballot_sync(unsigned, int);
void __syncwarp();
void __syncthreads();
template <typename T>
T __shfl_sync(unsigned, T, int);
template <typename T>
T __shfl_up_sync(unsigned, T, int);
template <typename T>
T __shfl_down_sync(unsigned, T, int);
template <typename T>
T atomicAdd(T *, T);
