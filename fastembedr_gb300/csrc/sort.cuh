// Block-level sorting primitive shared by the graph builders (t-SNE P, UMAP fuzzy graph).
#pragma once

#include <cuda_runtime.h>

namespace fe {

// Always-ascending bitonic network over `pw` (power of two) slots; compare(i, j) keeps the
// minimum at i. Slots at or beyond `len` hold +inf (explicitly in shared memory, virtually
// in global memory), which this formulation never moves below a real key.
template <bool kGlobal>
__device__ __forceinline__ void bitonic_sort(unsigned long long* a, int len, int pw) {
  for (int size = 2; size <= pw; size <<= 1) {
    const int half = size >> 1;
    for (int t = threadIdx.x; t < pw / 2; t += blockDim.x) {
      const int blk = t / half, off = t % half;
      const int i = blk * size + off, j = blk * size + size - 1 - off;
      if (!kGlobal || j < len) {
        const unsigned long long x = a[i], y = a[j];
        if (y < x) {
          a[i] = y;
          a[j] = x;
        }
      }
    }
    __syncthreads();
    for (int stride = half >> 1; stride > 0; stride >>= 1) {
      for (int t = threadIdx.x; t < pw / 2; t += blockDim.x) {
        const int blk = t / stride, off = t % stride;
        const int i = blk * 2 * stride + off, j = i + stride;
        if (!kGlobal || j < len) {
          const unsigned long long x = a[i], y = a[j];
          if (y < x) {
            a[i] = y;
            a[j] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Ascending sort of 32 E keys held by a warp, lane l holding positions l E .. l E + E - 1: the same
// always-ascending network with strides below E inside a lane and the others by shuffles.
template <int E>
__device__ __forceinline__ void warp_sort(unsigned long long (&a)[E], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * E; size <<= 1) {
#pragma unroll
    for (int step = size >> 1; step > 0; step >>= 1) {
      // first step of a size: partner = position ^ (size - 1); then position ^ step
      const int x = step == (size >> 1) ? size - 1 : step;
      const int lx = x / E, ix = x % E;
      if (lx == 0) {
#pragma unroll
        for (int i = 0; i < E; ++i) {
          const int j = i ^ ix;
          if (j > i) {
            const unsigned long long u = a[i], v = a[j];
            a[i] = u < v ? u : v;
            a[j] = u < v ? v : u;
          }
        }
      } else {
        const bool low = (lane & (1 << (31 - __clz(lx)))) == 0;
        unsigned long long b[E];
#pragma unroll
        for (int i = 0; i < E; ++i) b[i] = __shfl_xor_sync(0xffffffffu, a[i ^ ix], lx);
#pragma unroll
        for (int i = 0; i < E; ++i) a[i] = ((a[i] < b[i]) == low) ? a[i] : b[i];
      }
    }
  }
}

}  // namespace fe
