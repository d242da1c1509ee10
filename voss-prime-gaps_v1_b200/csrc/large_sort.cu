// large_sort.cu — the large-gap list in ascending position order, sorted on the device.
//
// Tiles append large gaps in completion order; the API returns them by position.  The list is
// sorted where it lies: keys (positions, of which only the bits below the range's end vary)
// with the records' indices through CUB's device radix sort, then one gather.  For the 389,279
// records of [1, 10^12] this replaces ~9 ms of host sorting after the copy.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include "voss_internal.h"

namespace voss {

__global__ void large_keys_kernel(const LargeGapDev* __restrict__ in, uint32_t n, unsigned long long* __restrict__ keys,
                                  uint32_t* __restrict__ idx) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    keys[i] = in[i].position;
    idx[i] = i;
  }
}

__global__ void large_gather_kernel(const LargeGapDev* __restrict__ in, const uint32_t* __restrict__ idx, uint32_t n,
                                    LargeGapDev* __restrict__ out) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = in[idx[i]];
}

// Lists of up to kSmallSort records, in the stream behind the tiles and before the host knows how
// many there are: block b of G places the records of the b-th G-th of [lo, hi).  It goes over all positions once,
// counts those below its part and lists those in it (a 148th of the records of a whole list: gaps lie
// evenly over a range), ranks the list against itself and writes each record to its place.  A part with more
// records than the list holds is taken in pieces, halved until one fits; the positions are distinct, so that
// ends.  A list cut short at `cap` holds what the first tiles found, nearly all of it in a few parts: 10,000
// of the 2.2e6 gaps >= 200 of 2e11 integers take one block 0.43 ms, beside 34 ms of tiles.
// Bound by the latency of its reads, n per block from L2, where ranking every record against all n was
// bound by n^2 compares: with the launch's other closing work 17.4 us for 10,602 records, 47.9 before,
// 17.2 us for 15,826, 64.4 before, 11.4 us for 308, 15.1 before.  One launch and no second round trip
// instead of nine launches after one; beyond 16,384 records the radix sort.
constexpr int kRankBlock = 1024;
constexpr uint32_t kRankList = 2048;

__global__ void __launch_bounds__(kRankBlock, 1)
large_rank_kernel(const LargeGapDev* __restrict__ in, const uint32_t* __restrict__ count, uint32_t cap,
                  unsigned long long lo, unsigned long long hi, LargeGapDev* __restrict__ out) {
  __shared__ unsigned long long s_key[kRankList];
  __shared__ uint32_t s_idx[kRankList];
  __shared__ uint32_t s_below, s_listed;
  const uint32_t n = *count < cap ? *count : cap;
  if (n > kSmallSort) return;
  const unsigned long long span = hi - lo, width = span / gridDim.x + 1ull, b = blockIdx.x;
  unsigned long long from = lo + min(b * width, span);
  const unsigned long long end = lo + min((b + 1) * width, span);
  unsigned long long piece = end - from;
  while (from < end) {
    unsigned long long to = from + min(piece, end - from);
    while (true) {
      __syncthreads();
      if (threadIdx.x == 0) s_below = s_listed = 0;
      __syncthreads();
      uint32_t below = 0;
#pragma unroll 4
      for (uint32_t k = threadIdx.x; k < n; k += kRankBlock) {
        const unsigned long long p = in[k].position;
        below += p < from;
        if (p >= from && p < to) {
          const uint32_t at = atomicAdd(&s_listed, 1u);
          if (at < kRankList) {
            s_key[at] = p;
            s_idx[at] = k;
          }
        }
      }
      below = __reduce_add_sync(0xFFFFFFFFu, below);
      if (threadIdx.x % 32 == 0 && below) atomicAdd(&s_below, below);
      __syncthreads();
      if (s_listed <= kRankList || to - from < 2ull) break;
      piece = (to - from) / 2ull;
      to = from + piece;
    }
    const uint32_t m = min(s_listed, kRankList);
    for (uint32_t i = threadIdx.x; i < m; i += kRankBlock) {
      const unsigned long long mine = s_key[i];
      uint32_t rank = s_below;
#pragma unroll 8
      for (uint32_t k = 0; k < m; ++k) rank += s_key[k] < mine;
      out[rank] = in[s_idx[i]];
    }
    from = to;
    if (m < kRankList / 4) piece *= 2ull;
  }
}

int launch_large_sort_small(const LargeGapDev* in, const uint32_t* count, uint32_t cap, uint64_t lo, uint64_t hi,
                            LargeGapDev* out, int sm_count, void* stream) {
  large_rank_kernel<<<sm_count, kRankBlock, 0, (cudaStream_t)stream>>>(in, count, cap, lo, hi < lo ? lo : hi, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

size_t large_sort_temp_bytes(uint32_t n, int end_bit) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                  (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)n, 0, end_bit);
  return bytes;
}

int launch_large_sort(const LargeGapDev* in, uint32_t n, int end_bit, unsigned long long* keys, uint32_t* idx,
                      void* temp, size_t temp_bytes, LargeGapDev* out, int sm_count, void* stream) {
  if (n == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const uint32_t blocks = (n + 255) / 256;
  const int grid = (int)(blocks < (uint32_t)sm_count * 8 ? blocks : (uint32_t)sm_count * 8);
  // keys/idx hold 2n entries: [0, n) input, [n, 2n) sorted output
  large_keys_kernel<<<grid, 256, 0, s>>>(in, n, keys, idx);
  if (cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys, keys + n, idx, idx + n, (int)n, 0, end_bit, s) !=
      cudaSuccess)
    return -1;
  large_gather_kernel<<<grid, 256, 0, s>>>(in, idx + n, n, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace voss
