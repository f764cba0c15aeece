// Where the rows of a step's requests lie when the keys that its new tokens see are put side by side: requests entry0 ..
// one after another, each from the first key that its first new token sees, rounded down to a whole tile of 128
// positions, to its last token, rounded up.
#pragma once

#include "common.cuh"

namespace ccb {

constexpr int kDenseTile = 128;

__device__ __forceinline__ int dense_first_key(int pos0, int window) {
  return (pos0 - window + 1 > 0 ? pos0 - window + 1 : 0) & ~(kDenseTile - 1);
}

__device__ __forceinline__ int dense_rows(const int* cu_q, const int* pos0, int e, int window) {
  const int end = pos0[e] + cu_q[e + 1] - cu_q[e];
  return ((end + kDenseTile - 1) & ~(kDenseTile - 1)) - dense_first_key(pos0[e], window);
}

// The first row of request e; all lanes of a warp call this together and get the same answer.
__device__ __forceinline__ int dense_base(const int* cu_q, const int* pos0, int entry0, int e, int window, int lane) {
  int sum = 0;
  for (int i = entry0 + lane; i < e; i += 32) sum += dense_rows(cu_q, pos0, i, window);
  return __reduce_add_sync(0xffffffffu, sum);
}

}  // namespace ccb
