// Compaction of the active positions of a schedule, and the inverse of its order.
#pragma once

#include "sweep_device.cuh"

namespace swk {

constexpr int kScanThreads = 1024;

// ---------------------------------------------------------------------------------------
// exclusive scan of the chunk counts in place (one block); the total goes to *count
static __global__ void __launch_bounds__(kScanThreads) k_compact_scan(uint32_t* chunk, uint32_t n, uint32_t* count) {
  __shared__ uint32_t warp_sum[kScanThreads / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < n; base += kScanThreads) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < n ? chunk[i] : 0u;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    uint32_t wbase = 0, total = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) {
      const uint32_t ws = warp_sum[w];
      if ((uint32_t)w < warp) wbase += ws;
      total += ws;
    }
    if (i < n) chunk[i] = carry + wbase + x - v;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) *count = carry;
}

// ---------------------------------------------------------------------------------------
// Compaction of a sparse level from a bitmap: the inverse of the schedule order gives
// each active cell's D positions, which set one bit each; a count / scan / scatter over
// the bitmap words then yields the active positions in schedule order.  The work is the
// active cells' tasks plus one pass over N*D/8 bytes.

static __global__ void k_invert_order(const uint32_t* order, uint32_t total, uint32_t* pos_of_task) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < total; p += gridDim.x * blockDim.x)
    pos_of_task[order[p]] = p;
}

static __global__ void k_mark_active(const uint8_t* level, int cur, uint32_t n, int D, uint32_t Np,
                              const uint32_t* pos_of_task, uint32_t* bitmap) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    if (level[c] < cur) continue;
    for (int d = 0; d < D; ++d) {
      const uint32_t p = pos_of_task[(size_t)d * Np + c];
      atomicOr(bitmap + (p >> 5), 1u << (p & 31u));
    }
  }
}

constexpr int kBitsThreads = 256;  // one bitmap word per thread, kBitsThreads words per chunk

static __global__ void __launch_bounds__(kBitsThreads) k_bits_count(const uint32_t* bitmap, uint32_t words, uint32_t* chunk) {
  const uint32_t w = blockIdx.x * kBitsThreads + threadIdx.x;
  uint32_t n = w < words ? __popc(bitmap[w]) : 0u;
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  __shared__ uint32_t ws[kBitsThreads / 32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = 0;
    for (int i = 0; i < kBitsThreads / 32; ++i) s += ws[i];
    chunk[blockIdx.x] = s;
  }
}

static __global__ void __launch_bounds__(kBitsThreads) k_bits_scatter(const uint32_t* bitmap, uint32_t words,
                                                               const uint32_t* chunk, uint32_t* act) {
  const uint32_t w = blockIdx.x * kBitsThreads + threadIdx.x;
  uint32_t bits = w < words ? bitmap[w] : 0u;
  // block-exclusive prefix of the per-thread counts
  __shared__ uint32_t ws[kBitsThreads / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t mine = __popc(bits);
  uint32_t x = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  uint32_t base = 0;
  for (uint32_t i = 0; i < warp; ++i) base += ws[i];
  uint32_t o = chunk[blockIdx.x] + base + x - mine;
  while (bits) {
    const int k = __ffs(bits) - 1;
    act[o++] = w * 32u + (uint32_t)k;
    bits &= bits - 1;
  }
}

}  // namespace swk
