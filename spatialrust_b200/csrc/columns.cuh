// columns.cuh -- a chain's result columns into the caller's device memory.
#pragma once

#include "plans.cuh"

namespace srcu {

constexpr int TAKE_MAX = 32;
constexpr int TAKE_THREADS = 256;
constexpr int TAKE_UNROLL = 4;  // 16-byte loads in flight per thread

// Columns of 32-bit words: `words` words per row, one row per voxel or point.
struct TakeColumns {
  const uint32_t *src[TAKE_MAX];
  uint32_t *dst[TAKE_MAX];
  uint32_t words[TAKE_MAX];
  uint32_t count;
};

// Copies the first rows of every column, *rows of them or, with rows null, count;
// blockIdx.y names the column.  A chain's row count is read on the device, so the copies follow the chain without
// waiting for the host to learn it, and one launch takes them all, where a copy
// per column after the wait left the GPU idle for its launch latency ten times
// (call and fetch of a 131k-point frame 250 -> 212 us; of a 2M-point scan with
// seven columns 578 -> 478 us).  Memory-bound at large sizes, hence the 16-byte
// accesses where both ends are aligned.
__global__ void __launch_bounds__(TAKE_THREADS) k_take_columns(const Control *ctl, TakeColumns t,
                                                               const unsigned long long *rows,
                                                               unsigned long long count) {
  if (rows && ctl->status) return;
  const uint32_t c = blockIdx.y;
  const uint32_t *src = t.src[c];
  uint32_t *dst = t.dst[c];
  const uint64_t n = (rows ? *rows : count) * t.words[c];
  const uint64_t stride = uint64_t(gridDim.x) * TAKE_THREADS;
  uint64_t i = blockIdx.x * uint64_t(TAKE_THREADS) + threadIdx.x;
  uint64_t done = 0;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
    const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
    uint4 *d4 = reinterpret_cast<uint4 *>(dst);
    const uint64_t n4 = n / 4;
    uint64_t k = i;
    for (; k + (TAKE_UNROLL - 1) * stride < n4; k += TAKE_UNROLL * stride) {
      uint4 v[TAKE_UNROLL];
#pragma unroll
      for (int q = 0; q < TAKE_UNROLL; ++q) v[q] = __ldcs(s4 + k + q * stride);
#pragma unroll
      for (int q = 0; q < TAKE_UNROLL; ++q) __stcs(d4 + k + q * stride, v[q]);
    }
    for (; k < n4; k += stride) d4[k] = s4[k];
    done = n4 * 4;
  }
  for (uint64_t k = done + i; k < n; k += stride) dst[k] = src[k];
}

}  // namespace srcu
