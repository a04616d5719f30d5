// The part of the CUDA device language that the windowed network's headers use,
// for a host compiler: the qualifiers, the vector types, and barriers and shared
// memory on the threads of tests/win_network.cpp.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

#define __device__
#define __global__
#define __host__
#define __shared__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))

struct alignas(16) uint4 {
    unsigned x, y, z, w;
};
struct alignas(8) int2 {
    int x, y;
};
struct dim3 {
    unsigned x = 1, y = 1, z = 1;
};
inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return uint4{x, y, z, w}; }
inline int2 make_int2(int x, int y) { return int2{x, y}; }
inline int min(int a, int b) { return std::min(a, b); }
inline int max(int a, int b) { return std::max(a, b); }
template <class T>
T __ldcs(const T* p) {
    return *p;
}
template <class T>
void __stcs(T* p, T v) {
    *p = v;
}

// barriers of the simulated threads
void __syncwarp();
void __syncthreads();
int __syncthreads_and(int v);

// named by code that the host build does not run
extern dim3 threadIdx, blockIdx, gridDim, blockDim;
template <class T>
T __shfl_xor_sync(unsigned, T v, int) {
    return v;
}
template <class T>
T __shfl_down_sync(unsigned, T v, int) {
    return v;
}
template <class T>
T __shfl_sync(unsigned, T v, int) {
    return v;
}
inline int __all_sync(unsigned, int v) { return v; }
inline size_t __cvta_generic_to_shared(const void* p) { return reinterpret_cast<size_t>(p); }
inline int atomicAdd(int* p, int v) { return (*p += v) - v; }
