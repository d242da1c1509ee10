// mr_kernels.cu — deterministic Miller-Rabin and gap proofs on sm_100a.
//
// Result-for-result equal to the reference verifier src/verify_cpp.cpp:
//   is_prime_u64 (:38-57): n < 2 -> composite; for each base B in {2,...,37}: n == B -> prime,
//   B | n -> composite; then the strong-probable-prime test to every base.
//   verify_gap (:59-93): both ends prime, then every interior integer must be marked by the
//   interval sieve (evens, then odd multiples of the odd base primes q <= isqrt(p_after)).
//
// The verdicts are exact for every 64-bit n, so they equal the reference's twelve strong
// probable-prime tests, which are exact below 2^64 too.  They come from trial division by 2..37, a
// strong probable-prime test to base 2 and, for its survivors, an extra strong Lucas test (Baillie
// and Wagstaff 1980; Grantham 2001: the smallest P >= 3 with (P^2 - 4 | n) = -1, Q = 1): no
// composite below 2^64 passes both (checked over Feitsma's list of all base-2 pseudoprimes below
// 2^64; PARI's and FLINT's primality tests of 64-bit integers rest on the same fact).  The Lucas
// test costs two products per bit, the five to eleven further bases it replaces 1.5 each.
//
// Arithmetic, by the size of n:
//   n < 2^49: products mod n in double precision from exact fma halves (DMod): six operations of the
//             fp64 pipe, 9.96 products per cycle and SM measured;
//   others:   64-bit Montgomery multiplication with R = 2^64 (mul.lo/mul.hi on the integer pipe, no
//             128-bit division), 2.36 per cycle and SM.
// One kernel does all of it: candidates that trial division leaves open wait in per-warp queues by
// test and size, and each time a queue holds 32 they are tested together, a lane each.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <mutex>

#include "voss.h"

#include "voss_internal.h"

namespace voss {

// Divisibility of n by the odd bases B (index 0, for 2, is not used): n B^-1 mod 2^64 is at most
// floor((2^64-1)/B) exactly when B | n.  Constant-initialised: the tables come with the kernel's module, so that
// no launch on any stream can run ahead of an upload.
struct TrialTables {
  uint64_t inv[12], lim[12];
};

constexpr TrialTables make_trial_tables() {
  constexpr uint64_t bases[12] = {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37};
  TrialTables t{};
  for (int i = 1; i < 12; ++i) {
    uint64_t x = bases[i];  // its own inverse mod 2^3
    for (int k = 0; k < 5; ++k) x *= 2ull - bases[i] * x;
    t.inv[i] = x;
    t.lim[i] = ~0ull / bases[i];
  }
  return t;
}
__constant__ TrialTables c_trial = make_trial_tables();

struct Mont {
  uint64_t n, inv, ninv, one, mone;  // inv = n^-1, ninv = -n^-1 (mod 2^64); one = 2^64 mod n, mone = n - one
};

// a b / 2^64 mod n for a, b < n: with m = (a b) n^-1 mod 2^64 the low halves of a b and m n agree, so
// the quotient is the difference of the high halves, without a carry; one conditional addition.
__device__ __forceinline__ uint64_t mont_mul(uint64_t a, uint64_t b, const Mont& M) {
  const uint64_t lo = a * b;
  const uint64_t hi = __umul64hi(a, b);
  const uint64_t mh = __umul64hi(lo * M.inv, M.n);
  const uint64_t t = hi - mh;
  return hi < mh ? t + M.n : t;
}

// The same for n < 2^63 as a sum: with m = -(a b) n^-1 the low halves add up to 2^64 (or 0), and
// hi + mh + carry < 2n < 2^64 (2.36 products per cycle and SM against 2.22).
__device__ __forceinline__ uint64_t mont_mul_small(uint64_t a, uint64_t b, const Mont& M) {
  const uint64_t lo = a * b;
  const uint64_t hi = __umul64hi(a, b);
  const uint64_t m = lo * M.ninv;
  const uint64_t t = hi + __umul64hi(m, M.n) + (lo != 0 ? 1ull : 0ull);
  return t >= M.n ? t - M.n : t;
}

__device__ __forceinline__ uint64_t mod_add(uint64_t a, uint64_t b, uint64_t n) {
  const uint64_t s = a + b;
  return (s < a || s >= n) ? s - n : s;
}

// 2^64 mod n for odd n > 1.  For n >= 2^32 the quotient q* = floor(2^64 / n), 1 <= q* < 2^32,
// is estimated in double precision (relative error < 2^-51, so the estimate is off by at most 1)
// and lowered by one, but not below 1: then q* - 2 <= q <= q* and q >= 1, so 2^64 - q n is below
// 2^64, lies in [0, 3n), and at most two subtractions finish it.  Smaller n take the 64-bit
// integer remainder.
__device__ __forceinline__ uint64_t two64_mod(uint64_t n) {
  if (n < (1ull << 32)) return (0ull - n) % n;
  uint64_t q = (uint64_t)(18446744073709551616.0 / (double)n);
  q = q > 1 ? q - 1 : 1;
  uint64_t r = 0ull - q * n;  // 2^64 - q n
  if (r >= n) r -= n;
  if (r >= n) r -= n;
  return r;
}

__device__ __forceinline__ Mont mont_setup(uint64_t n) {
  Mont M;
  M.n = n;
  uint64_t x = n;  // inverse of n mod 2^3
#pragma unroll
  for (int i = 0; i < 5; ++i) x *= 2ull - n * x;
  M.inv = x;
  M.ninv = 0ull - x;
  M.one = two64_mod(n);  // R mod n
  M.mone = n - M.one;
  return M;
}

// Trial phase of is_prime_u64: 1 = prime, 0 = composite, -1 = undecided.
__device__ __forceinline__ int trial_phase(uint64_t n) {
  if (n < 2) return 0;  // (41^2 = 1681 is the smallest composite that stays undecided)
  if (n == 2) return 1;
  if ((n & 1ull) == 0) return 0;
#pragma unroll
  for (int i = 1; i < 12; ++i) {
    const uint64_t B = i == 1 ? 3 : i == 2 ? 5 : i == 3 ? 7 : i == 4 ? 11 : i == 5 ? 13 : i == 6 ? 17
                     : i == 7 ? 19 : i == 8 ? 23 : i == 9 ? 29 : i == 10 ? 31 : 37;
    if (n == B) return 1;
    if (n * c_trial.inv[i] <= c_trial.lim[i]) return 0;
  }
  if (n < 1681) return 1;
  return -1;
}

// ---- products mod n in double precision -------------------------------------------------------
// For odd n in [1681, 2^49) and integers |a|, |b| < n (a doubled factor below 2n is allowed too): an
// integer r = a b (mod n) with |r| < n, all values exact in doubles.  h = a b rounded and l = a b - h
// (fma, exact); q = h / n rounded to an integer by adding 1.5 * 2^52 in the same rounding; h - q n is
// an integer below 2^53, so the fma that computes it is exact.  |q - h/n| <= 1/2 + |h/n| 2^-53 (the
// rounding of 1/n) and |l| <= |h| 2^-53 <= (|a b| / n) n 2^-53, so with |a b| <= 2 B^2 n^2 and n < 2^49
// |r| <= (1/2 + B^2 / 4) n: B = 0.59 reproduces itself.
constexpr uint64_t kDModEnd = 1ull << 49;
struct DMod {
  double n, inv;
};

__device__ __forceinline__ DMod dmod_setup(uint64_t n) {
  DMod M;
  M.n = (double)n;
  M.inv = __drcp_rn(M.n);
  return M;
}

__device__ __forceinline__ double dmod_mul(double a, double b, const DMod& M) {
  constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
  const double h = a * b;
  const double l = __fma_rn(a, b, -h);
  const double q = __fma_rn(h, M.inv, kRound) - kRound;
  return __fma_rn(-q, M.n, h) + l;
}

// ---- strong probable-prime test to base 2 -----------------------------------------------------
// Warp-uniform: every lane runs the same number of squarings (the warp's longest exponent and
// largest r) and keeps its verdict in a flag.  Early exits inside these loops let the lanes of a
// warp drift apart and never reconverge (measured: 2.8 active lanes per instruction).
struct OddPart {
  uint64_t d;  // m = d 2^r
  int r, top_w, r_w;  // top_w, r_w: the warp's longest d (index of the top bit) and largest r
};

__device__ __forceinline__ OddPart odd_part(uint64_t m) {
  OddPart E;
  E.r = __ffsll((long long)m) - 1;
  E.d = m >> E.r;
  E.top_w = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)(63 - __clzll(E.d)));
  E.r_w = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)E.r);
  return E;
}

__device__ __forceinline__ bool sprp2(const DMod& M, const OddPart& E) {
  // the top five bits of the exponent at once: 2^e <= 2^31 reduced by one product
  int b = E.top_w > 4 ? E.top_w - 4 : 0;
  double x = dmod_mul((double)(1u << (uint32_t)(E.d >> b)), 1.0, M);
  for (--b; b >= 0; --b) {
    const double y = x + x;
    x = dmod_mul(x, ((E.d >> b) & 1ull) ? y : x, M);
  }
  bool ok = (x == 1.0) | (x == -1.0);
  for (int j = 0; j < E.r_w - 1; ++j) {
    x = dmod_mul(x, x, M);
    ok |= (j < E.r - 1) & (x == -1.0);
  }
  return ok;
}

// kSmallN: every lane's n < 2^63 (mont_mul_small).
template <bool kSmallN>
__device__ __forceinline__ uint64_t mont_product(uint64_t a, uint64_t b, const Mont& M) {
  return kSmallN ? mont_mul_small(a, b, M) : mont_mul(a, b, M);
}

template <bool kSmallN>
__device__ __forceinline__ bool sprp2(const Mont& M, const OddPart& E) {
  uint64_t x = M.one;
  for (int b = E.top_w; b >= 0; --b) {
    x = mont_product<kSmallN>(x, x, M);
    const uint64_t y = mod_add(x, x, M.n);
    x = ((E.d >> b) & 1ull) ? y : x;
  }
  bool ok = (x == M.one) | (x == M.mone);
  for (int j = 0; j < E.r_w - 1; ++j) {
    x = mont_product<kSmallN>(x, x, M);
    ok |= (j < E.r - 1) & (x == M.mone);
  }
  return ok;
}

// ---- extra strong Lucas test --------------------------------------------------------------------
// Jacobi symbol (a | n) for odd n and 0 < a < 2^32.
__device__ inline int jacobi(uint32_t a, uint64_t n) {
  int j = 1;
  int z = __ffs((int)a) - 1;
  a >>= z;
  if ((z & 1) && ((n & 7) == 3 || (n & 7) == 5)) j = -j;
  if ((a & 3) == 3 && (n & 3) == 3) j = -j;
  uint32_t b = (uint32_t)(n % a);  // (a | n) = +-(n mod a | a)
  while (b) {
    z = __ffs((int)b) - 1;
    b >>= z;
    if ((z & 1) && ((a & 7) == 3 || (a & 7) == 5)) j = -j;
    if ((a & 3) == 3 && (b & 3) == 3) j = -j;
    const uint32_t t = a % b;
    a = b;
    b = t;
  }
  return a == 1 ? j : 0;
}

// The smallest P >= 3 with (P^2 - 4 | n) = -1 for odd n without prime factors up to 37; 0 when n is
// found composite on the way (a perfect square, for which there is none, or a common factor).
// P^2 - 4 = 5, 12, 21, 32, 45, 60, 77, 96, 117, ...: while the symbols of the primes up to 13 are
// all +1, only 5, 3, 7, 2, 11, 13, 17, 19 bring a new one, at P = 3, 4, 5, 6, 9, 11, 15, 17.
__device__ __forceinline__ uint32_t lucas_p(uint64_t n) {
  const uint32_t m = (uint32_t)(n % 4849845ull);  // 3 * 5 * 7 * 11 * 13 * 17 * 19
  const uint32_t n3 = (uint32_t)(n >> 1) & 1u;    // n = 3 (mod 4): (q | n) = -(n | q) for q = 3 (mod 4)
  const uint32_t n8 = (uint32_t)n & 7u;
  // bit n mod q of the masks: non-residues of q
  const uint32_t b5 = (0xCu >> (m % 5u)) & 1u, b3 = ((0x4u >> (m % 3u)) & 1u) ^ n3;
  const uint32_t b7 = ((0x68u >> (m % 7u)) & 1u) ^ n3, b2 = (n8 == 3u || n8 == 5u) ? 1u : 0u;
  const uint32_t b11 = ((0x5C4u >> (m % 11u)) & 1u) ^ n3, b13 = (0x9E4u >> (m % 13u)) & 1u;
  const uint32_t b17 = (0x5CE8u >> (m % 17u)) & 1u, b19 = ((0x4F50Cu >> (m % 19u)) & 1u) ^ n3;
  const uint32_t minus = b5 | b3 << 1 | b7 << 2 | b2 << 3 | b11 << 4 | b13 << 5 | b17 << 6 | b19 << 7;
  if (minus) return (uint32_t)(0x110F0B0906050403ull >> (8 * (__ffs((int)minus) - 1))) & 0xFFu;
  const uint64_t s = (uint64_t)sqrt((double)n);
  for (uint64_t t = s > 0 ? s - 1 : 0; t <= s + 1 && t <= 0xFFFFFFFFull; ++t)
    if (t * t == n) return 0;
  for (uint32_t P = 20;; ++P) {  // n is no square: half of all symbols are -1
    const int j = jacobi(P * P - 4u, n);
    if (j == -1) return P;
    if (j == 0) return 0;
  }
}

// n + 1 = d 2^s: passes if U_d = 0 and V_d = +-2, or V_{d 2^r} = 0 for some 0 <= r < s - 1 (mod n).
// The ladder holds (V_k, V_{k+1}): V_{2k} = V_k^2 - 2, V_{2k+1} = V_k V_{k+1} - P, two products per
// bit.  U_d = 0 <=> 2 V_{d+1} = P V_d, i.e. V_{d+1} = P or -P beside V_d = 2 or -2.  All lanes start from
// (V_0, V_1) = (2, P), which leading zero bits leave alone, so they share one trip count.
__device__ __forceinline__ bool lucas(const DMod& M, const OddPart& E, uint32_t P) {
  const double p = (double)P;
  double v = 2.0, w = p;
  for (int b = E.top_w; b >= 0; --b) {
    const bool one = (E.d >> b) & 1ull;
    const double t = dmod_mul(v, w, M) - p;
    const double x = one ? w : v;
    const double y = dmod_mul(x, x, M) - 2.0;
    v = one ? t : y;
    w = one ? y : t;
  }
  bool ok = (v == 2.0 && w == p) | (v == -2.0 && w == -p);
  ok |= (E.r > 1) & (v == 0.0);
  for (int j = 1; j < E.r_w - 1; ++j) {
    v = dmod_mul(v, v, M) - 2.0;
    ok |= (j < E.r - 1) & (v == 0.0);
  }
  return ok;
}

__device__ __forceinline__ uint64_t mod_sub(uint64_t a, uint64_t b, uint64_t n) {
  return a >= b ? a - b : a - b + n;
}

template <bool kSmallN>
__device__ __forceinline__ bool lucas(const Mont& M, const OddPart& E, uint32_t P) {
  const uint64_t n = M.n, two = mod_add(M.one, M.one, n);
  uint64_t p = 0;  // P R mod n by doubling
  for (int b = 31 - __clz((int)P); b >= 0; --b) {
    p = mod_add(p, p, n);
    if ((P >> b) & 1u) p = mod_add(p, M.one, n);
  }
  uint64_t v = two, w = p;
  for (int b = E.top_w; b >= 0; --b) {
    const bool one = (E.d >> b) & 1ull;
    const uint64_t t = mod_sub(mont_product<kSmallN>(v, w, M), p, n);
    const uint64_t x = one ? w : v;
    const uint64_t y = mod_sub(mont_product<kSmallN>(x, x, M), two, n);
    v = one ? t : y;
    w = one ? y : t;
  }
  bool ok = (v == two && w == p) | (v == n - two && w == n - p);
  ok |= (E.r > 1) & (v == 0);
  for (int j = 1; j < E.r_w - 1; ++j) {
    v = mod_sub(mont_product<kSmallN>(v, v, M), two, n);
    ok |= (j < E.r - 1) & (v == 0);
  }
  return ok;
}

// The two tests of a warp's 32 candidates, all of one size class (kDouble: n < kDModEnd).
template <bool kDouble>
__device__ __forceinline__ bool test_base2(uint64_t n) {
  const OddPart E = odd_part(n - 1);
  if (kDouble) return sprp2(dmod_setup(n), E);
  const Mont M = mont_setup(n);
  return __all_sync(0xFFFFFFFFu, n < (1ull << 63)) ? sprp2<true>(M, E) : sprp2<false>(M, E);
}

template <bool kDouble>
__device__ __forceinline__ bool test_lucas(uint64_t n) {
  const uint32_t P = lucas_p(n);
  __syncwarp();
  const OddPart E = odd_part(n + 1);  // n + 1 < 2^64: 2^64 - 1 has small factors
  bool ok;
  if (kDouble) {
    ok = lucas(dmod_setup(n), E, P);
  } else {
    const Mont M = mont_setup(n);
    ok = __all_sync(0xFFFFFFFFu, n < (1ull << 63)) ? lucas<true>(M, E, P) : lucas<false>(M, E, P);
  }
  return ok && P != 0;
}

// The same as calls: one copy of each test instead of one at every place that drains a queue.
template <bool kDouble>
__device__ __noinline__ bool call_base2(uint64_t n) {
  return test_base2<kDouble>(n);
}

template <bool kDouble>
__device__ __noinline__ bool call_lucas(uint64_t n) {
  return test_lucas<kDouble>(n);
}

// Trial division for every candidate (a lane per candidate); the undecided wait in the warp's
// shared-memory queues, one per size class for the base-2 test and one for the Lucas test of its
// survivors, and each time a queue holds 32 they are tested together.  Lanes whose candidate is
// decided early, and short exponents beside long ones, would otherwise leave most of the warp idle
// (13 of 32 lanes active per instruction when each lane ran its own test).
// Bound by the pipe of the products: 5e6 primes below 10^12 take 0.50 ms (two tests in double
// precision; 3.6 ms with six Montgomery tests each), 4,000,001 random odd 64-bit numbers 0.34 ms
// (0.77 ms with up to twelve bases and the survivors in a work list for a second kernel), 1000 of
// them 24 us (123 us).  Eight blocks per SM were chosen with the tests inlined (four resident: two waves, the second
// evening out what the warps of the first happen to find).  Large batches run them as calls now (below), five
// resident, and 8 is no longer the best: 4, 5, 8, 10, 15 and 16 per SM take 334, 339, 341, 321, 329 and 333 us
// for these 64-bit numbers, 525, 516, 492, 499, 488 and 487 us for the primes.
constexpr int kMrBlock = 256;
constexpr int kMrBlocksPerSm = 8;
constexpr int kMrQueue = 64;  // at most 31 waiting + 32 arriving

// Take up to 32 entries from the queue's front; lanes beyond `take` repeat lane 0's.
__device__ __forceinline__ uint32_t queue_take(uint32_t* q, uint32_t& nq, uint32_t lane, bool& live) {
  __syncwarp();
  const uint32_t take = nq < 32u ? nq : 32u;
  live = lane < take;
  const uint32_t i = q[live ? lane : 0u];
  __syncwarp();
  if (lane + 32u < nq) q[lane] = q[lane + 32u];
  nq -= take;
  __syncwarp();
  return i;
}

__device__ __forceinline__ void queue_add(uint32_t* q, uint32_t& nq, uint32_t lane, uint32_t i, bool add) {
  const unsigned m = __ballot_sync(0xFFFFFFFFu, add);
  if (add) q[nq + __popc(m & ((1u << lane) - 1u))] = i;
  nq += __popc(m);
}

struct MrQueues {  // of one size class
  uint32_t *base2, *lucas;
  uint32_t n_base2, n_lucas;
};

template <bool kDouble, bool kCalls>
__device__ __forceinline__ void drain_lucas(const uint64_t* __restrict__ cand, uint8_t* __restrict__ out, MrQueues& Q,
                                            uint32_t lane) {
  bool live;
  const uint32_t i = queue_take(Q.lucas, Q.n_lucas, lane, live);
  const bool ok = kCalls ? call_lucas<kDouble>(cand[i]) : test_lucas<kDouble>(cand[i]);
  if (live) out[i] = ok ? 1 : 0;
}

template <bool kDouble, bool kCalls>
__device__ __forceinline__ void drain_base2(const uint64_t* __restrict__ cand, uint8_t* __restrict__ out, MrQueues& Q,
                                            uint32_t lane) {
  bool live;
  const uint32_t i = queue_take(Q.base2, Q.n_base2, lane, live);
  const bool ok = kCalls ? call_base2<kDouble>(cand[i]) : test_base2<kDouble>(cand[i]);
  if (live && !ok) out[i] = 0;
  queue_add(Q.lucas, Q.n_lucas, lane, i, live && ok);
  if (Q.n_lucas >= 32u) drain_lucas<kDouble, kCalls>(cand, out, Q, lane);
}

// kCalls: for batches that give every block more than one pass.  Inlined, the tests stand at four
// places each, and a block whose candidates lie on both sides of 2^49 runs through more code than the
// instruction cache holds (ncu: 2.4 warps waiting for an instruction per issue); as calls there is one
// copy, and five blocks fit an SM.  10^7 candidates, half of them below 10^12 and half 64-bit: 1031 ->
// 920 us, 10^6 of them 150 -> 138, 4*10^6 of 48 bits 134 -> 125; 5*10^6 primes below 10^12 490 -> 488 and
// 4*10^6 64-bit ones 327 -> 335; but 1000 candidates, in calls, 22.7 -> 25.2 us.
template <bool kCalls>
__global__ void __launch_bounds__(kMrBlock, kCalls ? 5 : 1) mr_kernel(const uint64_t* __restrict__ cand, uint64_t count,
                                                                      uint8_t* __restrict__ out) {
  __shared__ uint32_t s_q[kMrBlock / 32][4][kMrQueue];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  MrQueues qd = {s_q[warp][0], s_q[warp][1], 0, 0}, qm = {s_q[warp][2], s_q[warp][3], 0, 0};
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + 32u * warp; base < count; base += stride) {
    const uint64_t i = base + lane;
    bool open = false, dbl = false;
    if (i < count) {
      const uint64_t n = cand[i];
      const int t = trial_phase(n);
      if (t >= 0) out[i] = (uint8_t)t;
      else {
        open = true;
        dbl = n < kDModEnd;
      }
    }
    queue_add(qd.base2, qd.n_base2, lane, (uint32_t)i, open && dbl);
    queue_add(qm.base2, qm.n_base2, lane, (uint32_t)i, open && !dbl);
    if (qd.n_base2 >= 32u) drain_base2<true, kCalls>(cand, out, qd, lane);
    if (qm.n_base2 >= 32u) drain_base2<false, kCalls>(cand, out, qm, lane);
  }
  // What is left in the queues (up to 31 each) is put together over the block, so that the last
  // tests run on full warps: at 4,000,001 candidates a warp sees 422 and leaves half a warp of
  // candidates for each test.
  __shared__ uint32_t s_rest[4][kMrBlock / 32 * 32];
  __shared__ uint32_t s_n[4];
  if (threadIdx.x < 4) s_n[threadIdx.x] = 0;
  __syncthreads();
  auto put = [&](int k, const uint32_t* q, uint32_t nq) {
    __syncwarp();  // the entries come from other lanes (queue_add); its ballot does not order shared memory
    uint32_t at = 0;
    if (lane == 0 && nq) at = atomicAdd(&s_n[k], nq);
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    if (lane < nq) s_rest[k][at + lane] = q[lane];
  };
  put(0, qd.base2, qd.n_base2);
  put(1, qm.base2, qm.n_base2);
  qd.n_base2 = qm.n_base2 = 0;
  __syncthreads();
  // base 2: the block's warps take 32 at a time; survivors go to the warp's Lucas queue (31 + 32 fit)
  auto take = [&](int k, uint32_t c, uint32_t* q, uint32_t& nq) {
    const uint32_t n = s_n[k], first = 32u * c;
    if (first >= n) return false;
    nq = min(32u, n - first);
    if (lane < nq) q[lane] = s_rest[k][first + lane];
    return true;
  };
  constexpr uint32_t kWarps = kMrBlock / 32;
  for (uint32_t c = warp; take(0, c, qd.base2, qd.n_base2); c += kWarps) drain_base2<true, kCalls>(cand, out, qd, lane);
  for (uint32_t c = warp; take(1, c, qm.base2, qm.n_base2); c += kWarps)
    drain_base2<false, kCalls>(cand, out, qm, lane);
  put(2, qd.lucas, qd.n_lucas);
  put(3, qm.lucas, qm.n_lucas);
  __syncthreads();
  for (uint32_t c = warp; take(2, c, qd.lucas, qd.n_lucas); c += kWarps) drain_lucas<true, kCalls>(cand, out, qd, lane);
  for (uint32_t c = kWarps - 1 - warp; take(3, c, qm.lucas, qm.n_lucas); c += kWarps)
    drain_lucas<false, kCalls>(cand, out, qm, lane);
}

// Gap proofs: one warp per gap.  Interior integers are split over the lanes; an interior odd
// integer is marked by the reference's sieve iff it has an odd prime factor q <= isqrt(p_after),
// i.e. iff it is composite or itself a prime <= isqrt(p_after).
__device__ __forceinline__ uint64_t isqrt64(uint64_t x) {
  uint64_t s = (uint64_t)sqrt((double)x);
  if (s > 0xFFFFFFFFull) s = 0xFFFFFFFFull;
  while (s * s > x) --s;
  while (s < 0xFFFFFFFFull && (s + 1) * (s + 1) <= x) ++s;
  return s;
}

// Endpoints of every gap, [2g] = p_after - gap (as the reference: u64 wrap-around), [2g+1] = p_after.
__global__ void gap_ends_kernel(const uint64_t* __restrict__ p_after, const int32_t* __restrict__ gap,
                                uint64_t count, uint64_t* __restrict__ ends) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < count; g += stride) {
    const uint64_t pa = p_after[g];
    ends[2 * g] = pa - (uint64_t)(int64_t)gap[g];
    ends[2 * g + 1] = pa;
  }
}

constexpr int kProveBlock = 256;
constexpr uint32_t kProveChunk = 256;  // interior odd integers examined per round (list capacity)

// Interior proofs, one warp per gap, after the endpoints have been tested (end_ok).  Per round of
// kProveChunk odd interior integers: trial division by the bases 3..37 on all lanes, the
// undecided integers above isqrt(p_after) are appended to a per-warp list in shared memory, and
// the list is tested 32 at a time by a warp-uniform base-2 strong probable-prime test; only
// integers passing it (primes, or base-2 strong pseudoprimes) take the Lucas test.
__global__ void __launch_bounds__(kProveBlock) prove_interior_kernel(const uint64_t* __restrict__ p_after,
                                                                     const int32_t* __restrict__ gap, uint64_t count,
                                                                     const uint8_t* __restrict__ end_ok,
                                                                     uint8_t* __restrict__ ok) {
  __shared__ uint64_t s_list[kProveBlock / 32][kProveChunk];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  uint64_t* list = s_list[wib];
  const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t g = (uint64_t)blockIdx.x * (blockDim.x >> 5) + wib; g < count; g += warps) {
    const uint64_t pa = p_after[g];
    const int32_t gp = gap[g];
    const uint64_t pb = pa - (uint64_t)(int64_t)gp;
    bool res = end_ok[2 * g] && end_ok[2 * g + 1];
    if (res && gp >= 2) {
      if ((pb & 1ull) == 0) {
        res = false;  // p_before = 2: the even-index marking leaves interior 4 unmarked
      } else {
        const uint64_t sq = isqrt64(pa);
        const uint64_t n_odd = (uint64_t)(gp - 2) / 2;  // odd integers pb+2 .. pa-2
        bool bad = false;
        for (uint64_t k0 = 0; k0 < n_odd && !bad; k0 += kProveChunk) {
          const uint64_t k1 = n_odd - k0 < kProveChunk ? n_odd : k0 + kProveChunk;
          uint32_t n_list = 0;
          bool small_prime = false;
          for (uint64_t kb = k0; kb < k1; kb += 32) {  // warp-uniform trip count
            const uint64_t k = kb + lane;
            int t = 0;
            uint64_t v = 0;
            if (k < k1) {
              v = pb + 2 + 2 * k;
              if (v > sq) t = trial_phase(v);  // 1: a base prime, 0: has a factor <= 37, -1: undecided
            }
            small_prime |= (t == 1);
            const unsigned m = __ballot_sync(0xFFFFFFFFu, t < 0);
            if (t < 0) list[n_list + (uint32_t)__popc(m & ((1u << lane) - 1u))] = v;
            n_list += (uint32_t)__popc(m);
          }
          __syncwarp();
          bad = __any_sync(0xFFFFFFFFu, small_prime);
          for (uint32_t b0 = 0; b0 < n_list && !bad; b0 += 32) {
            const bool live = b0 + lane < n_list;
            const uint64_t v = list[live ? b0 + lane : b0];  // idle lanes shadow the first entry
            const bool dbl = __all_sync(0xFFFFFFFFu, v < kDModEnd);
            const bool prp = dbl ? test_base2<true>(v) : test_base2<false>(v);
            if (__any_sync(0xFFFFFFFFu, prp)) {  // idle lanes have a live lane's verdict
              const bool prime = (dbl ? test_lucas<true>(v) : test_lucas<false>(v)) && prp;
              bad = __any_sync(0xFFFFFFFFu, prime);
            }
          }
          __syncwarp();
        }
        res = !bad;
      }
    }
    if (lane == 0) ok[g] = res ? 1 : 0;
  }
}

int launch_mr(const uint64_t* d_n, uint64_t count, uint8_t* d_out, void* stream, int sm_count) {
  if (count == 0) return 0;
  if (count > 0xFFFFFFFFull) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  const uint64_t want = (count + kMrBlock - 1) / kMrBlock;
  const uint64_t most = (uint64_t)sm_count * kMrBlocksPerSm;
  if (want > most) mr_kernel<true><<<(int)most, kMrBlock, 0, s>>>(d_n, count, d_out);
  else mr_kernel<false><<<(int)want, kMrBlock, 0, s>>>(d_n, count, d_out);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_prove_gaps(const uint64_t* d_p_after, const int32_t* d_gap, uint64_t count, uint8_t* d_ok,
                      uint64_t* d_ends, uint8_t* d_ends_ok, void* stream, int sm_count) {
  if (count == 0) return 0;
  if (count > 0x7FFFFFFFull) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  // 1. both endpoints of every gap through the Miller-Rabin kernel
  const uint64_t eg = (count + 255) / 256;
  gap_ends_kernel<<<(int)(eg < (uint64_t)sm_count * 8 ? eg : (uint64_t)sm_count * 8), 256, 0, s>>>(d_p_after, d_gap,
                                                                                                   count, d_ends);
  if (launch_mr(d_ends, 2 * count, d_ends_ok, stream, sm_count)) return -1;
  // 2. interiors
  const uint64_t want = (count + (kProveBlock / 32) - 1) / (kProveBlock / 32);
  const int grid = (int)(want < (uint64_t)sm_count * 8 ? want : (uint64_t)sm_count * 8);
  prove_interior_kernel<<<grid, kProveBlock, 0, s>>>(d_p_after, d_gap, count, d_ends_ok, d_ok);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Peak rates of the modular products on this device: independent squaring chains, every lane
// active, no branches and no memory traffic.  The roofline denominators of the primality
// kernels, which spend their time in the same products (one figure per variant: doubles below 2^49,
// Montgomery moduli below and above 2^63).
constexpr int kMulmodChains = 8;
constexpr int kMulmodIters = 2048;
constexpr int kMulmodBlock = 256;

template <bool kSmallN>
__global__ void __launch_bounds__(kMulmodBlock) mulmod_probe_kernel(uint64_t nbase, uint64_t* sink) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t n = nbase | (tid << 1) | 1ull;  // an odd modulus per thread
  const Mont M = mont_setup(n);
  uint64_t x[kMulmodChains];
#pragma unroll
  for (int c = 0; c < kMulmodChains; ++c) x[c] = (M.one >> 1) + (uint64_t)c + 1ull;  // < n
#pragma unroll 1
  for (int i = 0; i < kMulmodIters; ++i) {
#pragma unroll
    for (int c = 0; c < kMulmodChains; ++c) x[c] = kSmallN ? mont_mul_small(x[c], x[c], M) : mont_mul(x[c], x[c], M);
  }
  uint64_t acc = 0;
#pragma unroll
  for (int c = 0; c < kMulmodChains; ++c) acc ^= x[c];
  if (acc == 1ull) sink[0] = acc;  // keeps the chains live; practically never taken
}

__global__ void __launch_bounds__(kMulmodBlock) dmod_probe_kernel(uint64_t nbase, uint64_t* sink) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const DMod M = dmod_setup(nbase | (tid << 1) | 1ull);
  double x[kMulmodChains];
#pragma unroll
  for (int c = 0; c < kMulmodChains; ++c) x[c] = (double)(nbase >> 2) + (double)c;
#pragma unroll 1
  for (int i = 0; i < kMulmodIters; ++i) {
#pragma unroll
    for (int c = 0; c < kMulmodChains; ++c) x[c] = dmod_mul(x[c], x[c], M);
  }
  double acc = 0;
#pragma unroll
  for (int c = 0; c < kMulmodChains; ++c) acc += x[c];
  if (acc == 1.0) sink[0] = 1;  // as above
}

static int probe_products(void (*kernel)(uint64_t, uint64_t*), uint64_t nbase, int sm_count, cudaStream_t s,
                          uint64_t* sink, double* per_s) {
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kMulmodBlock, 0) != cudaSuccess || occ < 1) return -1;
  const int grid = sm_count * occ;  // one full wave
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return -1;
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return -1;
  }
  kernel<<<grid, kMulmodBlock, 0, s>>>(nbase, sink);  // warm-up
  const int reps = 3;
  cudaEventRecord(e0, s);
  for (int r = 0; r < reps; ++r) kernel<<<grid, kMulmodBlock, 0, s>>>(nbase, sink);
  cudaEventRecord(e1, s);
  const cudaError_t st = cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (st != cudaSuccess || ms <= 0) return -1;
  *per_s = (double)grid * kMulmodBlock * kMulmodChains * kMulmodIters * reps / (ms * 1e-3);
  return 0;
}

int probe_mulmod(int sm_count, void* stream, double* full_per_s, double* small_per_s, double* dbl_per_s) {
  cudaStream_t s = (cudaStream_t)stream;
  uint64_t* sink = nullptr;
  if (cudaMalloc(&sink, sizeof(uint64_t)) != cudaSuccess) return -1;
  int rc = 0;
  if (full_per_s) rc |= probe_products(mulmod_probe_kernel<false>, 3ull << 62, sm_count, s, sink, full_per_s);
  if (small_per_s) rc |= probe_products(mulmod_probe_kernel<true>, 1ull << 62, sm_count, s, sink, small_per_s);
  if (dbl_per_s) rc |= probe_products(dmod_probe_kernel, kDModEnd >> 1, sm_count, s, sink, dbl_per_s);
  cudaFree(sink);
  return rc;
}

}  // namespace voss

// =====================================================================================
// Miller-Rabin without any allocation (voss_mr_verify_noalloc).
//
// Some callers cannot allocate device memory at call time: a process whose device memory is
// already reserved by another allocator (a framework's caching allocator or a memory pool),
// where cudaMalloc would fail or fragment that pool, and request paths of long-running
// services, where cudaMalloc/cudaFree would synchronize the device and stall other streams.
// The regular entry points allocate (the context at creation, per-call buffers on growth); this
// one needs no context and no device memory of its own.
// =====================================================================================
namespace voss {

constexpr uint64_t kNoAllocMaxCount = 1ull << 22;  // candidates per call

static std::mutex g_noalloc_mu;
static int g_noalloc_sms[64];  // SM count per device ordinal

}  // namespace voss

namespace voss_detail {
int set_error(int code, const char* msg);
}

extern "C" VOSS_API int voss_mr_verify_noalloc(const uint64_t* d_n, uint64_t count, uint8_t* d_is_prime,
                                               void* stream) {
  using namespace voss;
  char msg[160];
  if (count == 0) return VOSS_OK;
  if (!d_n || !d_is_prime) return voss_detail::set_error(VOSS_ERR_ARG, "NULL device pointer");
  if (count > kNoAllocMaxCount) {
    snprintf(msg, sizeof(msg), "count %llu exceeds the no-allocation limit of %llu candidates per call",
             (unsigned long long)count, (unsigned long long)kNoAllocMaxCount);
    return voss_detail::set_error(VOSS_ERR_ARG, msg);
  }
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return voss_detail::set_error(VOSS_ERR_NODEV, "no current CUDA device");
  int sms = 0;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_sms[dev]) {
      int n = 0;
      if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
        return voss_detail::set_error(VOSS_ERR_CUDA, "cannot read the SM count");
      g_noalloc_sms[dev] = n;
    }
    sms = g_noalloc_sms[dev];
  }
  if (launch_mr(d_n, count, d_is_prime, stream, sms) != 0) {
    snprintf(msg, sizeof(msg), "Miller-Rabin launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    return voss_detail::set_error(VOSS_ERR_CUDA, msg);
  }
  return VOSS_OK;
}
