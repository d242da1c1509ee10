// short_iv.cu — short intervals at high starts by Miller-Rabin instead of the sieve.
//
// Sieving [lo, hi) reduces lo modulo every base prime up to isqrt(hi - 1): at hi = 10^16 that
// is 5.76e6 reductions however short the interval, and at 10^18 50.8e6.  Testing the
// interval's wheel integers (coprime to 30) with the deterministic primality kernel costs
// about 30 products per integer instead, so voss_sieve_intervals sends an interval
// here when its base primes outnumber mr_route times its length.  The verdicts are exact for
// every n < 2^64 (mr_kernels.cu), so the statistics are the ones the sieve gives: primes >= 7 of
// [lo, hi), their gap histogram (bin g/2), first and last prime, and the first maximal gap.
#include <cuda_runtime.h>

#include <cstdint>

#include "voss.h"
#include "voss_internal.h"

namespace voss {

namespace {

constexpr int kShortBlock = 256;
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ uint64_t wheel_value(const ShortInterval& I, uint32_t j) {
  const uint32_t J = I.j0 + j;
  return I.base + 30ull * (J >> 3) + ((kW30Packed >> (8u * (J & 7u))) & 0xFFu);
}

// The intervals are worked on in segments of kShortSeg candidates, a block each, so that one long
// interval fills the GPU as well as many short ones.  Segment b belongs to the last interval with
// seg_begin <= b; every interval has at least one.
__device__ __forceinline__ uint32_t interval_of(const ShortInterval* __restrict__ iv, uint32_t n_iv, uint32_t b) {
  uint32_t lo = 0, hi = n_iv;
  while (hi - lo > 1u) {
    const uint32_t mid = (lo + hi) >> 1;
    if (iv[mid].seg_begin <= b) lo = mid; else hi = mid;
  }
  return lo;
}

// The wheel integers of every short interval, in order, at cand[cand_off ...]; each interval's first
// segment clears its histogram.
__global__ void __launch_bounds__(kShortBlock) short_cand_kernel(const ShortInterval* __restrict__ iv, uint32_t n_iv,
                                                                 uint32_t n_seg, uint64_t* __restrict__ cand,
                                                                 voss_interval_stats* __restrict__ out) {
  for (uint32_t b = blockIdx.x; b < n_seg; b += gridDim.x) {
    const ShortInterval I = iv[interval_of(iv, n_iv, b)];
    const uint64_t j0 = (uint64_t)(b - I.seg_begin) * kShortSeg;
    const uint32_t j1 = (uint32_t)min(j0 + kShortSeg, (uint64_t)I.n_cand);
    for (uint32_t j = (uint32_t)j0 + threadIdx.x; j < j1; j += blockDim.x) cand[I.cand_off + j] = wheel_value(I, j);
    if (b == I.seg_begin)
      for (uint32_t i = threadIdx.x; i < (uint32_t)VOSS_IHIST; i += blockDim.x) out[I.out_index].gap_hist[i] = 0;
  }
}

__device__ __forceinline__ void add_gap(unsigned long long* hist, uint64_t g, uint32_t& over) {
  if (g < 2ull * VOSS_IHIST)
    atomicAdd(hist + (g >> 1), 1ull);
  else
    ++over;
}

__device__ __forceinline__ void longer_gap(uint32_t& g, unsigned long long& lo, uint32_t g2, unsigned long long lo2) {
  if (g2 > g || (g2 == g && lo2 < lo)) {  // ties go to the smaller lower prime, as in the sieve path
    g = g2;
    lo = lo2;
  }
}

// A block's totals of (count, over, first prime, last prime, longest gap), to thread 0.
struct Totals {
  uint32_t cnt, over, g;
  unsigned long long first, last, lo;  // ~0 (first, lo) or 0 (last) when there is none
};

__device__ __forceinline__ void add_totals(Totals& a, const Totals& b) {
  a.cnt += b.cnt;
  a.over += b.over;
  a.first = b.first < a.first ? b.first : a.first;
  a.last = b.last > a.last ? b.last : a.last;
  longer_gap(a.g, a.lo, b.g, b.lo);
}

__device__ __forceinline__ void block_totals(Totals& t, Totals* s_tot) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    Totals o;
    o.cnt = __shfl_down_sync(kFull, t.cnt, d);
    o.over = __shfl_down_sync(kFull, t.over, d);
    o.g = __shfl_down_sync(kFull, t.g, d);
    o.first = __shfl_down_sync(kFull, t.first, d);
    o.last = __shfl_down_sync(kFull, t.last, d);
    o.lo = __shfl_down_sync(kFull, t.lo, d);
    add_totals(t, o);
  }
  if (lane == 0) s_tot[warp] = t;
  __syncthreads();
  if (threadIdx.x == 0)
    for (uint32_t w = 1; w < kShortBlock / 32; ++w) add_totals(t, s_tot[w]);
}

// A block per segment: its candidates are split into one contiguous chunk per thread, walked in
// order; the gap into each chunk comes from the last prime of the nearest earlier chunk (an
// exclusive max-scan: primes increase with the chunk index).
__global__ void __launch_bounds__(kShortBlock) short_seg_kernel(const ShortInterval* __restrict__ iv, uint32_t n_iv,
                                                                uint32_t n_seg, const uint8_t* __restrict__ ok,
                                                                voss_interval_stats* __restrict__ out,
                                                                ShortSegment* __restrict__ seg) {
  __shared__ uint32_t hist[VOSS_IHIST];
  __shared__ unsigned long long w_scan[kShortBlock / 32];
  __shared__ Totals s_tot[kShortBlock / 32];
  constexpr uint32_t kPer = kShortSeg / kShortBlock;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  for (uint32_t b = blockIdx.x; b < n_seg; b += gridDim.x) {
    const ShortInterval I = iv[interval_of(iv, n_iv, b)];
    for (uint32_t i = tid; i < (uint32_t)VOSS_IHIST; i += kShortBlock) hist[i] = 0;
    __syncthreads();
    const uint64_t j0 = (uint64_t)(b - I.seg_begin) * kShortSeg + kPer * tid;
    uint32_t mask = 0;  // verdicts of the chunk
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k)
      if (j0 + k < I.n_cand && ok[I.cand_off + j0 + k]) mask |= 1u << k;
    Totals t = {(uint32_t)__popc(mask), 0, 0, ~0ull, 0, ~0ull};
    auto count_gap = [&](uint64_t lo, uint64_t hi) {
      const uint64_t g = hi - lo;
      if (g < 2ull * VOSS_IHIST) atomicAdd(hist + (g >> 1), 1u);
      else ++t.over;
      longer_gap(t.g, t.lo, (uint32_t)g, lo);
    };
    for (uint32_t m = mask; m; m &= m - 1u) {
      const uint64_t v = wheel_value(I, (uint32_t)j0 + (uint32_t)__ffs((int)m) - 1u);
      if (t.last) count_gap(t.last, v);
      else t.first = v;
      t.last = v;
    }
    unsigned long long incl = t.last;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long u = __shfl_up_sync(kFull, incl, d);
      if (lane >= (uint32_t)d && u > incl) incl = u;
    }
    if (lane == 31) w_scan[warp] = incl;
    __syncthreads();
    unsigned long long ex = __shfl_up_sync(kFull, incl, 1);
    if (lane == 0) ex = 0;
    for (uint32_t w = 0; w < warp; ++w) ex = w_scan[w] > ex ? w_scan[w] : ex;
    if (mask && ex) count_gap(ex, t.first);
    block_totals(t, s_tot);
    if (tid == 0) seg[b] = ShortSegment{t.first, t.last, t.lo, t.g, t.cnt, t.over, 0};
    __syncthreads();
    unsigned long long* h = reinterpret_cast<unsigned long long*>(out[I.out_index].gap_hist);
    for (uint32_t i = tid; i < (uint32_t)VOSS_IHIST; i += kShortBlock)
      if (hist[i]) atomicAdd(h + i, (unsigned long long)hist[i]);
    __syncthreads();  // hist and the warp scratch are reused by the next segment
  }
}

// A block per interval: its segments put together, and the gaps between them.
__global__ void __launch_bounds__(kShortBlock) short_stats_kernel(const ShortInterval* __restrict__ iv,
                                                                  uint32_t n_iv, const ShortSegment* __restrict__ seg,
                                                                  voss_interval_stats* __restrict__ out) {
  __shared__ Totals s_tot[kShortBlock / 32];
  for (uint32_t b = blockIdx.x; b < n_iv; b += gridDim.x) {
    const ShortInterval I = iv[b];
    voss_interval_stats* s = out + I.out_index;
    const uint32_t n = short_segments(I.n_cand);
    Totals t = {0, 0, 0, ~0ull, 0, ~0ull};
    for (uint32_t i = threadIdx.x; i < n; i += kShortBlock) {
      const ShortSegment S = seg[I.seg_begin + i];
      add_totals(t, Totals{S.count, S.over, S.max_gap, S.first, S.last, S.max_gap_lo});
      if (!S.count) continue;
      unsigned long long before = 0;  // last prime of the nearest earlier segment that has one
      for (uint32_t k = i; k && !before;) before = seg[I.seg_begin + --k].last;
      if (before) {
        add_gap(reinterpret_cast<unsigned long long*>(s->gap_hist), S.first - before, t.over);
        longer_gap(t.g, t.lo, (uint32_t)(S.first - before), before);
      }
    }
    block_totals(t, s_tot);
    if (threadIdx.x == 0) {
      s->lo = 0;
      s->hi = 0;
      s->prime_count = t.cnt;
      s->first_prime = t.cnt ? t.first : 0;
      s->last_prime = t.last;
      s->max_gap = t.g;
      s->max_gap_lo = t.g ? t.lo : 0;
      s->gap_overflow = t.over;
    }
    __syncthreads();  // s_tot is reused by the next interval
  }
}

}  // namespace

int launch_short_intervals(const ShortInterval* d_iv, uint32_t n_iv, uint32_t n_seg, uint64_t n_cand,
                           uint64_t* d_cand, uint8_t* d_ok, ShortSegment* d_seg, voss_interval_stats* d_out,
                           int sm_count, void* stream) {
  if (n_iv == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const uint32_t most = (uint32_t)sm_count * 8u;
  const uint32_t grid = n_seg < most ? n_seg : most;
  short_cand_kernel<<<grid, kShortBlock, 0, s>>>(d_iv, n_iv, n_seg, d_cand, d_out);
  if (n_cand && launch_mr(d_cand, n_cand, d_ok, stream, sm_count)) return -1;
  short_seg_kernel<<<grid, kShortBlock, 0, s>>>(d_iv, n_iv, n_seg, d_ok, d_out, d_seg);
  short_stats_kernel<<<n_iv < most ? n_iv : most, kShortBlock, 0, s>>>(d_iv, n_iv, d_seg, d_out);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace voss
