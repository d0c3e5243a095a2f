// One row of at most 8192 columns spread over a group of threads: the layout and the sum that the RMSNorm kernels
// share, so that a norm gives the same bits wherever it runs (on its own, or behind a split-K reduction).
//
// A thread owns 16-byte vectors (8 bf16) c = tid + group * i. One vector a thread up to 4096 columns: a row of 2048 is
// 256 threads, which keeps eight rows in flight on an SM, needs few registers and, for the handful of rows of a decode step, spreads a
// row over eight warps instead of one.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace b200 {

struct RmsShape {
  int group;  // threads of a row, a multiple of 32
  int vpt;    // vectors of a thread: 1 or 2
};

__host__ __device__ inline RmsShape rms_shape(int H) {
  const int nvec = H >> 3;
  const int vpt = nvec <= 512 ? 1 : 2;
  return {((nvec + vpt - 1) / vpt + 31) / 32 * 32, vpt};
}

constexpr int kRmsMaxWarps = 16;

// Sums of ROWS numbers over the `group` threads of slot `y` (a barrier of its own each); `part`: the slot's ROWS *
// kRmsMaxWarps floats of shared memory, which the caller does not reuse before the group's next barrier but one.
template <int ROWS>
__device__ __forceinline__ void rms_group_sums(float (&v)[ROWS], float* part, int tid, int group, int y) {
#pragma unroll
  for (int k = 0; k < ROWS; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if (group == 32) return;
  if ((tid & 31) == 0)
#pragma unroll
    for (int k = 0; k < ROWS; ++k) part[k * kRmsMaxWarps + (tid >> 5)] = v[k];
  asm volatile("bar.sync %0, %1;" ::"r"(1 + y), "r"(group) : "memory");
  const int nw = group >> 5;
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    float s = 0.f;
    for (int w = 0; w < nw; ++w) s += part[k * kRmsMaxWarps + w];
    v[k] = s;
  }
}

__device__ __forceinline__ float rms_group_sum(float v, float* part, int tid, int group, int y) {
  float a[1] = {v};
  rms_group_sums<1>(a, part, tid, group, y);
  return a[0];
}

}  // namespace b200
