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
// many there are: every record counts the positions below its own (they are distinct) and is written
// to that place.  A block ranks 64 records; its four warp pairs count in a quarter of the keys each,
// 1024 keys at a time in shared memory.  One launch and no second round trip instead of nine launches
// after one (a bitonic sort in one block took 8 us for 300 records and 50 us for 2000, on its
// barriers); beyond 16,384 records the radix sort is the faster one.
constexpr int kRankBlock = 256, kRankRecords = 64;
constexpr uint32_t kRankKeys = 1024;  // per round, a quarter of them per warp pair

__global__ void __launch_bounds__(kRankBlock) large_rank_kernel(const LargeGapDev* __restrict__ in,
                                                                const uint32_t* __restrict__ count, uint32_t cap,
                                                                LargeGapDev* __restrict__ out) {
  __shared__ __align__(16) unsigned long long s_key[kRankKeys];
  __shared__ uint32_t s_rank[kRankRecords];
  const uint32_t n = *count < cap ? *count : cap;
  const uint32_t r = threadIdx.x % kRankRecords, part = threadIdx.x / kRankRecords;
  const uint32_t first = kRankRecords * blockIdx.x;
  if (n > kSmallSort || first >= n) return;
  const LargeGapDev mine = in[min(first + r, n - 1)];
  if (threadIdx.x < kRankRecords) s_rank[threadIdx.x] = 0;
  uint32_t rank = 0;
  for (uint32_t base = 0; base < n; base += kRankKeys) {
    __syncthreads();
#pragma unroll
    for (uint32_t k = threadIdx.x; k < kRankKeys; k += kRankBlock)
      s_key[k] = base + k < n ? in[base + k].position : ~0ull;
    __syncthreads();
    const ulonglong2* keys = reinterpret_cast<const ulonglong2*>(s_key + part * (kRankKeys / 4));
#pragma unroll 8
    for (uint32_t k = 0; k < kRankKeys / 8; ++k) {
      const ulonglong2 x = keys[k];
      rank += (x.x < mine.position) + (x.y < mine.position);
    }
  }
  atomicAdd(&s_rank[r], rank);
  __syncthreads();
  if (part == 0 && first + r < n) out[s_rank[r]] = mine;
}

int launch_large_sort_small(const LargeGapDev* in, const uint32_t* count, uint32_t cap, LargeGapDev* out,
                            void* stream) {
  const uint32_t most = cap < kSmallSort ? cap : kSmallSort;
  large_rank_kernel<<<(most + kRankRecords - 1) / kRankRecords, kRankBlock, 0, (cudaStream_t)stream>>>(in, count, cap, out);
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
