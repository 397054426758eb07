// What a host compiler needs to read the device headers of cosmos_gb300/csrc (tests only): CUDA's
// qualifiers as nothing, and the few builtins their non-template functions name.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __host__
#define __global__
#define __shared__ static
#define __forceinline__ inline
#define __noinline__
#define __grid_constant__
#define __launch_bounds__(...)

inline double __longlong_as_double(long long x) {
    double d;
    memcpy(&d, &x, 8);
    return d;
}
inline long long __double_as_longlong(double x) {
    long long u;
    memcpy(&u, &x, 8);
    return u;
}
inline unsigned long long __ldcg(unsigned long long* p) { return *p; }
inline unsigned long long atomicMax(unsigned long long* p, unsigned long long) { return *p; }
inline int atomicOr(int* p, int v) {
    *p |= v;
    return 0;
}
inline void __syncthreads() {}
template <class T> T __shfl_xor_sync(unsigned, T v, int) { return v; }
struct HostIndex { unsigned x, y, z; };
static HostIndex threadIdx, blockIdx, blockDim, gridDim;
using std::isfinite;
