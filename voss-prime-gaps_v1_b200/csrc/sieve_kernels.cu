// sieve_kernels.cu — the sm_100a sieve-and-gap kernels.
//
// One persistent kernel (sieve_tiles_kernel) replaces the reference's per-segment pipeline
// memset -> graph of one sieve_w30_seg_kernel launch per base prime -> extract -> thrust::sort
// -> mod4 -> modq -> gaps (src/voss_v7_live.cu:120-312, 480-585).  Each CTA claims tiles of the
// wheel-30 bitmap from an atomic work counter and, for every tile, entirely in shared memory:
//   1. fill:     writes the tile pre-sieved by 7..31 from four periodic word-mask tables and
//                masks the interval's ends (the reference's cudaMemset + first-word patch, :496-500);
//   2. sieve:    clears the odd multiples of the base primes 37 <= p <= isqrt(hi-1)
//                (the reference's sieve_w30_seg_kernel, :120-143, one launch per prime):
//                  small primes  p <  tile_bytes/coop_div : one warp per prime, its hits as 32
//                                                            progressions that never share a bank,
//                  medium primes p <  walk bound          : one thread per prime, 8 residues,
//                                p <  p_large           : one thread per prime of one class mod
//                                                            30, its eight first hits and rounds,
//                  large primes  otherwise                 : one thread per prime, walking its
//                                                            multiples across the tile's span;
//   3. restore:  sets the bits of base primes lying in the tile (the reference starts each prime
//                at p^2, :452-466; here the p*1 hit is undone instead);
//   4. extract:  the residue classes for mod-4 and mod-q (:181-232) are counted by word (all
//                words w = c mod 1001 share their class slots); then each thread walks an equal
//                share of the tile's primes in order (ffs), its predecessor prime coming from a
//                block-wide max-scan of the chunks' last primes, and updates shared-memory
//                counters: the gap histogram (:278-280), the per-residue gap histogram (:282-287),
//                the large-gap list (:289-299) and the tile's maximal gap.  Primes never reach HBM.
// The gaps across tile seams and each interval's first/last prime and maximal gap come from
// tail_kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "voss.h"
#include "voss_internal.h"

namespace voss {

// The wheel tables are constant-initialised: they come with the kernels' module, so that no launch on any
// stream can run ahead of an upload.
template <class T, int N>
struct Table {
  T v[N];
};

constexpr uint32_t wheel_residue(int o) { return (uint32_t)(kW30Packed >> (8 * o)) & 0xFFu; }

// residue r (mod 30) -> wheel bit index, or -1 when gcd(r, 30) > 1.
constexpr Table<int8_t, 32> make_res_bit() {
  Table<int8_t, 32> t{};
  for (int r = 0; r < 32; ++r) t.v[r] = -1;
  for (int o = 0; o < 8; ++o) t.v[wheel_residue(o)] = (int8_t)o;
  return t;
}
constexpr Table<int8_t, 32> kResBit = make_res_bit();
__constant__ Table<int8_t, 32> c_res_bit = make_res_bit();

// [bi*8 + o]: for a prime p = 30a + b (b = W30[bi]) and multiplier residue w = W30[o],
// p*w = 30*(a*w + D) + W30[B] with D = floor(b*w/30), stored as D | (B << 5).
constexpr Table<uint8_t, 64> make_wheel_step() {
  Table<uint8_t, 64> t{};
  for (int i = 0; i < 64; ++i) {
    const uint32_t bw = wheel_residue(i / 8) * wheel_residue(i % 8);
    t.v[i] = (uint8_t)(bw / 30u | (uint32_t)kResBit.v[bw % 30u] << 5);
  }
  return t;
}
__constant__ Table<uint8_t, 64> c_wheel_step = make_wheel_step();

// Wheel walk of a prime p = 30a + W30[bi] over its multiples p*m with gcd(m, 30) = 1.
// [bi*30 + t]: t = (offset of the first multiple of p at or above a tile's start) mod 30 gives
// m mod 30 = t * p^-1 (mod 30); stored: (steps to the next m coprime to 30) | (its wheel index << 3).
constexpr Table<uint8_t, 240> make_walk_start() {
  Table<uint8_t, 240> t{};
  for (int bi = 0; bi < 8; ++bi) {
    uint32_t pinv = 1;
    while (wheel_residue(bi) * pinv % 30u != 1u) ++pinv;
    for (uint32_t k = 0; k < 30; ++k) {
      const uint32_t u = k * pinv % 30u;
      uint32_t adv = 0;
      while (kResBit.v[(u + adv) % 30u] < 0) ++adv;
      t.v[bi * 30 + (int)k] = (uint8_t)(adv | (uint32_t)kResBit.v[(u + adv) % 30u] << 3);
    }
  }
  return t;
}
__constant__ Table<uint8_t, 240> c_walk_start = make_walk_start();

// [bi*8 + j]: from m = 30c + W30[j] to the next coprime m, the byte index of p*m grows by
// a*gap_j + corr (gap_j = W30[j+1] - W30[j], W30[8] = 31); stored: .x = ~(1 << bit of p*m)
// (rotated left by 8 * (byte & 3) it is the clear mask of that byte's lane in its word; the
// funnel shift takes its count mod 32, so byte << 3 is that rotation),
// .y = gap_j | corr << 16.
constexpr Table<uint2, 64> make_walk_step() {
  Table<uint2, 64> t{};
  for (int bi = 0; bi < 8; ++bi)
    for (int j = 0; j < 8; ++j) {
      const uint32_t w = wheel_residue(bi), m = wheel_residue(j), next = j < 7 ? wheel_residue(j + 1) : 31u;
      t.v[bi * 8 + j].x = ~(1u << kResBit.v[w * m % 30u]);
      t.v[bi * 8 + j].y = (next - m) | (w * next / 30u - w * m / 30u) << 16;
    }
  return t;
}
__constant__ Table<uint2, 64> c_walk_step = make_walk_step();

// [bi*8 + j], for the primes that a tile takes by class: .x = D_j - D_{j-1} (D_j = floor(W30[bi] W30[j] / 30),
// D_{-1} = 0), .y = the bit of W30[bi] * W30[j].
constexpr Table<uint2, 64> make_cls_step() {
  Table<uint2, 64> t{};
  for (int bi = 0; bi < 8; ++bi)
    for (int j = 0; j < 8; ++j) {
      const uint32_t w = wheel_residue(bi), m = wheel_residue(j);
      t.v[bi * 8 + j].x = w * m / 30u - (j ? w * wheel_residue(j - 1) / 30u : 0u);
      t.v[bi * 8 + j].y = (uint32_t)kResBit.v[w * m % 30u];
    }
  return t;
}
__constant__ Table<uint2, 64> c_cls_step = make_cls_step();

__device__ __forceinline__ uint32_t w30(uint32_t o) {
  return (uint32_t)((kW30Packed >> (8u * o)) & 0xFFu);
}

// x mod p with m = floor((2^64-1)/p): q <= x/p < q + 3.
__device__ __forceinline__ uint32_t mod_barrett(uint64_t x, uint32_t p, uint64_t m) {
  uint64_t q = __umul64hi(x, m);
  uint64_t r = x - q * (uint64_t)p;
  if (r >= p) r -= p;
  if (r >= p) r -= p;
  return (uint32_t)r;
}

// x mod p for x < 2^53 and 8 <= p < 2^30 from the Barrett constant m = floor((2^64-1)/p), with
// xs = x * 2^-64 as a double (exact).  m rounded to double times xs is x/p within a relative
// 2^-53 (x/p < 2^50), so adding 2^52 in the same rounding (fma) leaves an integer q within 0.63
// of x/p in the low mantissa bits; x - q p then lies in (-p, 2p), which its low 32 bits hold.
__device__ __forceinline__ uint32_t mod_by_magic_fma(uint64_t x, double xs, uint32_t p, uint64_t m) {
  const double qd = __fma_rn(xs, __ull2double_rn(m), 4503599627370496.0);
  uint32_t r = (uint32_t)x - (uint32_t)__double2loint(qd) * p;
  r += (int32_t)r < 0 ? p : 0u;
  r -= r >= p ? p : 0u;
  return r;
}

// x mod p for x < 2^58 and 8 <= p < 2^24, with xd = x as a double and inv = 1/p rounded to double.
// Below 2^53 xd is exact and xd * inv is x/p within a relative 2^-53 (x/p < 2^50: 1/8), so the
// integer q that adding 2^52 in the same rounding leaves in the low mantissa bits is within 0.63 of
// x/p: the low 32 bits of x - q p are the remainder or the remainder less p.  Larger x go in two
// steps of that kind: (x >> 28) mod p, then the rest below 2^24 * 2^28.
__device__ __forceinline__ uint32_t mod_by_inv(uint64_t x, double xd, uint32_t p, double inv) {
  constexpr double kTwo52 = 4503599627370496.0;
  uint32_t r;
  if (x < (1ull << 53)) {
    r = (uint32_t)x - (uint32_t)__double2loint(__fma_rn(xd, inv, kTwo52)) * p;
  } else {
    const uint32_t h = (uint32_t)(x >> 28);
    uint32_t rh = h - (uint32_t)__double2loint(__fma_rn((double)h, inv, kTwo52)) * p;
    rh = min(rh, rh + p);
    const uint64_t y = ((uint64_t)rh << 28) | (x & ((1ull << 28) - 1));
    r = (uint32_t)y - (uint32_t)__double2loint(__fma_rn((double)y, inv, kTwo52)) * p;
  }
  return min(r, r + p);  // a negative remainder is a large unsigned
}

__device__ __forceinline__ uint64_t isqrt_u64(uint64_t x) {
  uint64_t s = (uint64_t)sqrt((double)x);
  if (s > 0xFFFFFFFFull) s = 0xFFFFFFFFull;
  while (s * s > x) --s;
  while (s < 0xFFFFFFFFull && (s + 1) * (s + 1) <= x) ++s;
  return s;
}

// number of table primes <= v
__device__ __forceinline__ uint32_t count_le(const uint32_t* pr, uint32_t n, uint64_t v) {
  if (v >= 0xFFFFFFFFull) return n;
  uint32_t lo = 0, hi = n, x = (uint32_t)v;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (pr[mid] <= x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// number of table primes < v
__device__ __forceinline__ uint32_t count_lt(const uint32_t* pr, uint32_t n, uint64_t v) {
  if (v == 0) return 0;
  return count_le(pr, n, v - 1);
}

// number of table primes <= v, found by the 32 lanes of a warp together: each round probes 32
// evenly spaced entries of the remaining range and keeps the slice between the last probe <= v
// and the first > v, so a table of n primes takes about log32(n) rounds of loads instead of
// log2(n) dependent ones.  Every lane returns the count.
__device__ __forceinline__ uint32_t count_le_warp(const uint32_t* pr, uint32_t n, uint64_t v, uint32_t lane) {
  if (v >= 0xFFFFFFFFull) return n;
  const uint32_t x = (uint32_t)v;
  uint32_t lo = 0, hi = n;  // the count lies in [lo, hi]
  while (hi - lo > 32u) {
    const uint32_t step = (hi - lo + 31u) >> 5;
    const uint32_t pos = lo + lane * step;
    const bool le = pos < hi && pr[pos] <= x;
    const uint32_t k = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, le));  // probes 0..k-1 are <= x
    const uint32_t nlo = k ? lo + (k - 1u) * step + 1u : lo;
    const uint32_t bound = lo + k * step;  // the first probe > x, when it exists
    if (bound < hi) hi = bound;
    lo = nlo;
  }
  const bool le = lo + lane < hi && pr[lo + lane] <= x;
  return lo + (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, le));
}

__device__ __forceinline__ uint32_t count_lt_warp(const uint32_t* pr, uint32_t n, uint64_t v, uint32_t lane) {
  return v == 0 ? 0u : count_le_warp(pr, n, v - 1, lane);
}

__device__ __forceinline__ uint32_t find_interval(const SieveArgs& a, uint32_t t) {
  if (a.tile_iv) return a.tile_iv[t];  // the launch's tile -> interval table
  uint32_t lo = 0, hi = a.n_intervals;  // largest i with tile_begin <= t
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (a.iv[mid].tile_begin <= t) lo = mid; else hi = mid;
  }
  return lo;
}

#ifdef VOSS_BOUNDS_CHECK
#define VOSS_SM_GUARD(idx, limit)             \
  if ((idx) >= (limit)) {                     \
    atomicOr(err, kErrBounds);                \
    return;                                   \
  }
#else
#define VOSS_SM_GUARD(idx, limit)
#endif

// The tile's bitmap in shared memory, words addressed by byte offset (a multiple of 4).  A clear
// that may fall outside goes to the lane's own word behind the tile instead of around a branch:
// shared-memory atomics are not predicated, and the divergence region of a branch costs five
// instructions per clear (11.8 instructions against 6 for the hits of clear_class_primes).
struct TileBits {
  uint32_t* bm;
  uint32_t spare;  // byte offset of the lane's first word behind the tile (kSpareWords follow every tile)
  uint32_t nw;     // words of this tile
  uint32_t* err;

  __device__ __forceinline__ void clear(uint32_t off, uint32_t mask) const {
    VOSS_SM_GUARD(off >> 2, nw + kSpareWords)
    atomicAnd(reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(bm) + off), mask);
  }
  // Byte offset of byte x's word, or of the lane's k-th spare word (k < kSpareRows) when x >= 4 nw (an x
  // below zero is a large unsigned).  Clears that follow each other take different spare words: on one
  // word a warp's atomics in close succession serialise (the small primes' starts and ends, unrolled
  // by four, took 61k wavefronts per tile instead of 47k).
  __device__ __forceinline__ uint32_t word_or_spare(uint32_t x, int k) const {
    return __viaddmin_u32(spare, 128u * (uint32_t)k, x) & ~3u;
  }
  __device__ __forceinline__ void clear_word_or_spare(uint32_t off, uint32_t mask, int k) const {
    clear(__viaddmin_u32(spare, 128u * (uint32_t)k, off), mask);
  }
};

// The clear mask of bit `bit` of byte `byte`: ~1 rotated by 8 (byte mod 4) + bit (the funnel shift
// takes its count mod 32).
__device__ __forceinline__ uint32_t bit_mask(uint32_t byte, uint32_t bit) {
  return __funnelshift_l(0xFFFFFFFEu, 0xFFFFFFFEu, (byte << 3) + bit);
}

// Small primes, a warp per prime.  The prime's hits are 32 progressions of words, one per lane:
// residue o = lane mod 8, first hit u = lane / 8 of four; a lane's bytes are s_o + u p + 4 p k, so
// its byte lane, and with it the clear mask, is fixed and it advances by p words per step.  If lane
// l starts in word c_l, step k clears words c_l + p k: the banks of a step are those of step 0
// shifted, so lanes that collide once collide at every step.  As p is odd, p^-1 mod 32 turns banks
// into places phi_l = c_l p^-1 (mod 32) on a circle that every lane walks one place per step.  The
// lanes are sorted by phi (rank r_l) and lane l starts d_l = K + phi_l - r_l >= 0 steps late
// (K = max(r - phi)): at every step the 32 lanes then stand on 32 different places, i.e. in 32
// different banks, and each atomic instruction is a single wavefront.  The delays reach about 8
// steps (the spread of 32 uniform points around their ranks) next to the Lt / (4 p) steps of the
// prime.  Banks are the bound: an atomic of random banks takes 3.0 cycles of the SM's
// shared-memory pipe, a conflict-free one 1.0 (measured).  Per tile of 6.02e6 integers the small
// primes take 46k wavefronts; 4 lanes per residue at random banks from tile/512 on, with eight
// set-ups per prime below, took 81k.
__device__ __forceinline__ void clear_small_prime(const TileBits& T, uint32_t rec, const uint8_t* s_step,
                                                  uint32_t lane, uint32_t Lt) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  const uint32_t r = rec & 0x1FFFu, p = (rec >> 13) & 0x1FFFu, bi = rec >> 26;
  const uint32_t o = lane & 7u;
  const uint32_t e = s_step[bi * 8u + o];
  const uint32_t delta = (p / 30u) * w30(o) + (e & 31u);
  const uint32_t byte = (delta >= r ? delta - r : delta + p - r) + (lane >> 3) * p;
  const uint32_t mask = bit_mask(byte, e >> 5);
  const uint32_t word = byte >> 2;
  const uint32_t phi = (word * (p * (2u - p * p))) & 31u;  // p (2 - p^2) = p^-1 (mod 64) for odd p
  uint32_t rank = 0;
  unsigned eq = kFull;  // lanes whose phi agrees with mine in the bits looked at so far
#pragma unroll
  for (int b = 4; b >= 0; --b) {
    const bool one = (phi >> b) & 1u;
    const unsigned m = __ballot_sync(kFull, one);
    rank += one ? (uint32_t)__popc(eq & ~m) : 0u;
    eq &= one ? m : ~m;
  }
  rank += (uint32_t)__popc(eq & ((1u << lane) - 1u));
  const int K = __reduce_max_sync(kFull, (int)rank - (int)phi);
  const uint32_t late = (uint32_t)(K + (int)phi - (int)rank);
  // byte offsets of the words, negative before the lane's start (a large unsigned: the spare word);
  // Lt is a multiple of 4, so byte + 4 p k < Lt  <=>  4 (word + p k) < Lt
  uint32_t w = 4u * (word - p * late);
  const int step = 4 * (int)p;
  const int left = (int)(Lt - w);
  const int x_in = __reduce_max_sync(kFull, -(int)w);  // from here on every lane has started,
  const int x_out = __reduce_min_sync(kFull, left);    // up to here none has finished,
  const int x_end = __reduce_max_sync(kFull, left);    // and here all have
  int x = 0;
#pragma unroll 1
  for (; x < x_in; x += 4 * step) {
#pragma unroll
    for (int j = 0; j < 4; ++j, w += (uint32_t)step) T.clear_word_or_spare(w, mask, j);
  }
#pragma unroll 1
  for (const int x_8 = x_out - 7 * step; x < x_8; x += 8 * step) {
#pragma unroll
    for (int j = 0; j < 8; ++j, w += (uint32_t)step) T.clear(w, mask);
  }
#pragma unroll 1
  for (; x < x_end; x += 4 * step) {
#pragma unroll
    for (int j = 0; j < 4; ++j, w += (uint32_t)step) T.clear_word_or_spare(w, mask, j);
  }
}

// Clears bit `bit` of bytes byte, byte + p, byte + 2p, ... below Lt (p odd).  Four consecutive
// hits fall in the four distinct byte lanes of their words, and advancing all four by 4p bytes
// moves each by exactly p words, so the unrolled loop keeps four fixed masks and word offsets; the
// up to three hits that remain are predicated.
__device__ __forceinline__ void clear_progression(const TileBits& T, uint32_t byte, uint32_t p, uint32_t bit,
                                                  uint32_t Lt) {
  // the four hits' byte lanes are j0, j0 + p, j0 + 2p, j0 + 3p (mod 4): one lane up each time
  // for p = 1 (mod 4), one lane down for p = 3, so each mask is the previous one rotated by a byte
  const uint32_t b1 = byte + p, b2 = b1 + p, b3 = b2 + p;
  const uint32_t rot = (p & 2u) ? 24u : 8u;
  const uint32_t m0 = bit_mask(byte, bit), m1 = __funnelshift_l(m0, m0, rot), m2 = __funnelshift_l(m1, m1, rot);
  uint32_t w0 = byte & ~3u;
  const uint32_t d1 = (b1 & ~3u) - w0, d2 = (b2 & ~3u) - w0, step = 4u * p;
  if (b3 < Lt) {
    const uint32_t m3 = __funnelshift_l(m2, m2, rot);
    const uint32_t d3 = (b3 & ~3u) - w0;
    const uint32_t lim = Lt - (b3 - w0);  // b3 + 4pk < Lt  <=>  w0 + 4pk < lim
    do {
      T.clear(w0, m0);
      T.clear(w0 + d1, m1);
      T.clear(w0 + d2, m2);
      T.clear(w0 + d3, m3);
      w0 += step;
    } while (w0 < lim);
  }
  T.clear_word_or_spare(w0, m0, 0);
  T.clear_word_or_spare(w0 + d1, m1, 1);
  T.clear_word_or_spare(w0 + d2, m2, 2);
}

struct ClassStep {  // c_cls_step of one class
  uint32_t corr[8], bit[8];
};

// The multiples of 32 primes of one residue class mod 30 (p = 30a + W30[bi], a lane per prime, in
// ascending order, pmin the first lane's) in the tile: the first hits s_j of the eight
// progressions by additions from the remainder r of the tile's first byte (progression j holds
// the bytes = a W30[j] + D_j (mod p), and a step from j to j + 1 adds a (W30[j+1] - W30[j]) + corr_j),
// then rounds of eight predicated clears, each round one period p further.  For primes above the
// tile length one round does it.  The class is the warp's, so corr_j and the bits are the same
// for all lanes: nothing is looked up per hit, and nothing branches but the round loop.
// Bound by shared-memory wavefronts (3.6 per clear, random banks) and issue slots alike (84 and 77 % of
// their peaks): 343k warp instructions per tile near 10^12, against 451k of a walk from multiple to
// multiple whose steps depend on the lane's own class.  kOneRound (pmin >= Lt) clears each hit where
// it is found: 17.9 against 18.4 ms for the 10^11 integers below 10^12.
template <bool kOneRound>
__device__ __forceinline__ void clear_class_primes(const TileBits& T, uint32_t p, uint32_t r, uint32_t pmin,
                                                   const ClassStep& C, uint32_t Lt) {
  const uint32_t a = p / 30u, a2 = 2u * a, a4 = 2u * a2, a6 = a4 + a2;
  uint32_t x[8];        // the hits as bit indices: 8 times the byte plus the bit
  uint32_t t = 0u - r;  // in (-p, p)
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    constexpr uint32_t gap[8] = {1, 6, 4, 2, 4, 2, 4, 6};  // W30[j] - W30[j - 1]
    t += (gap[j] == 1 ? a : gap[j] == 2 ? a2 : gap[j] == 4 ? a4 : a6) + C.corr[j];
    const uint32_t s = __viaddmin_u32(t, p, t);  // t mod p: a negative t is a large unsigned
    if (kOneRound) T.clear(T.word_or_spare(s, j), bit_mask(s, C.bit[j]));
    else x[j] = 8u * s + C.bit[j];
  }
  if (kOneRound) return;
  const uint32_t period = 8u * p;
  for (uint32_t start = 0; start < Lt; start += pmin) {  // no hit of round start / pmin lies below byte start
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      T.clear(T.word_or_spare(x[j] >> 3, j), __funnelshift_l(0xFFFFFFFEu, 0xFFFFFFFEu, x[j]));
      x[j] += period;
    }
  }
}

// The word at shared-memory address p + 4 into x, and p on to it, if x is used up (zero): one
// predicated step, without a branch.
__device__ __forceinline__ void next_word_if_spent(uint32_t& x, uint32_t& p) {
  asm volatile(
      "{\n\t"
      ".reg .pred spent;\n\t"
      "setp.eq.u32 spent, %0, 0;\n\t"
      "@spent add.u32 %1, %1, 4;\n\t"
      "@spent ld.shared.u32 %0, [%1];\n\t"
      "}"
      : "+r"(x), "+r"(p)
      :
      : "memory");
}

__device__ __forceinline__ void sm_add(uint32_t* cnt, uint32_t idx, uint32_t* err) {
  VOSS_SM_GUARD(idx, (uint32_t)kSmCounters)
  atomicAdd(cnt + idx, 1u);
}

__device__ __forceinline__ void sm_add_n(uint32_t* cnt, uint32_t idx, uint32_t v, uint32_t* err) {
  VOSS_SM_GUARD(idx, (uint32_t)kSmCounters)
  atomicAdd(cnt + idx, v);
}

// Carry-save adder over bit planes: l = a ^ b ^ c, h = majority(a, b, c).
__device__ __forceinline__ void csa(uint32_t& h, uint32_t& l, uint32_t a, uint32_t b, uint32_t c) {
  const uint32_t u = a ^ b;
  h = (a & b) | (u & c);
  l = u ^ c;
}

// Swaps the bits of x selected by mask << s with the bits of y selected by mask (one step of an
// 8x8 bit-matrix transpose applied to the four byte lanes at once).
__device__ __forceinline__ void swap_bits(uint32_t& x, uint32_t& y, uint32_t mask, uint32_t s) {
  const uint32_t t = ((x >> s) ^ y) & mask;
  y ^= t;
  x ^= t << s;
}

// The residue-class counters of a tile's primes (k mod 28 and k mod 143 by wheel residue: every
// q of the reference's mod-4 and mod-q counts, voss_v7_live.cu:181-232), counted by word instead
// of by prime.  The slots of bit b of word w are 8 ((k28 + 4w) mod 28) + b and
// 8 ((k143 + 4w) mod 143) + b, and 4004 = 4 * 1001 is a multiple of 28 and of 143, so all words
// w = c (mod 1001) share their 32 slots in each block.  A thread takes the words of one class c
// and adds them column by column into six bit planes with carry-save adders (a column counts at
// most 63 words; shared memory holds tiles of at most about 52,000 words, at most 52 per class),
// transposes the planes into 32 byte-sized column counts and adds each column to its two slots:
// 64 shared-memory atomics per class instead of two per prime.  The planes are first rotated by
// the lane number, so lane l adds column (s + l) mod 32 at step s: the k mod 28 slots of a warp
// then lie in 32 distinct banks (8 (k28 + 4w) mod 32 is the same for every w), and the k mod 143
// slots as well once each lane's bytes are shifted by its own (k143 + 4c) mod 4.
template <int BLOCK>
__device__ __forceinline__ void class_counts_by_word(const uint32_t* bm, uint32_t nw, uint32_t k28,
                                                     uint32_t k143, uint32_t* cnt, uint32_t lane,
                                                     uint32_t* err) {
  for (uint32_t c = threadIdx.x; c < 1001u; c += BLOCK) {
    uint32_t p0 = 0, p1 = 0, p2 = 0, p3 = 0, p4 = 0, p5 = 0;
    uint32_t w = c;
    for (; w + 7u * 1001u < nw; w += 8u * 1001u) {  // eight words: three levels of adders
      uint32_t a1, a2, a3, a4, b1, b2, c1;
      csa(a1, p0, p0, bm[w], bm[w + 1001u]);
      csa(a2, p0, p0, bm[w + 2u * 1001u], bm[w + 3u * 1001u]);
      csa(b1, p1, p1, a1, a2);
      csa(a3, p0, p0, bm[w + 4u * 1001u], bm[w + 5u * 1001u]);
      csa(a4, p0, p0, bm[w + 6u * 1001u], bm[w + 7u * 1001u]);
      csa(b2, p1, p1, a3, a4);
      csa(c1, p2, p2, b1, b2);
      const uint32_t t3 = p3 & c1;
      p3 ^= c1;
      p5 ^= p4 & t3;
      p4 ^= t3;
    }
    for (; w < nw; w += 1001u) {  // the rest one word at a time
      const uint32_t x = bm[w];
      const uint32_t t0 = p0 & x;
      p0 ^= x;
      const uint32_t t1 = p1 & t0;
      p1 ^= t0;
      const uint32_t t2 = p2 & t1;
      p2 ^= t1;
      const uint32_t t3 = p3 & t2;
      p3 ^= t2;
      p5 ^= p4 & t3;
      p4 ^= t3;
    }
    // rotate: bit s of each plane becomes column (s + lane) mod 32
    p0 = __funnelshift_r(p0, p0, lane);
    p1 = __funnelshift_r(p1, p1, lane);
    p2 = __funnelshift_r(p2, p2, lane);
    p3 = __funnelshift_r(p3, p3, lane);
    p4 = __funnelshift_r(p4, p4, lane);
    p5 = __funnelshift_r(p5, p5, lane);
    // transpose each byte lane's 8x8 bit matrix (planes 6 and 7 are zero): afterwards byte n of
    // t_j is the count of rotated column 8n + j
    uint32_t t0 = p0, t1 = p1, t2 = p2, t3 = p3, t4 = p4, t5 = p5, t6 = 0, t7 = 0;
    swap_bits(t0, t4, 0x0F0F0F0Fu, 4);
    swap_bits(t1, t5, 0x0F0F0F0Fu, 4);
    swap_bits(t2, t6, 0x0F0F0F0Fu, 4);
    swap_bits(t3, t7, 0x0F0F0F0Fu, 4);
    swap_bits(t0, t2, 0x33333333u, 2);
    swap_bits(t1, t3, 0x33333333u, 2);
    swap_bits(t4, t6, 0x33333333u, 2);
    swap_bits(t5, t7, 0x33333333u, 2);
    swap_bits(t0, t1, 0x55555555u, 1);
    swap_bits(t2, t3, 0x55555555u, 1);
    swap_bits(t4, t5, 0x55555555u, 1);
    swap_bits(t6, t7, 0x55555555u, 1);
    const uint32_t tt[8] = {t0, t1, t2, t3, t4, t5, t6, t7};
    const uint32_t u28 = (k28 + 4u * c) % 28u, u143 = (k143 + 4u * c) % 143u;
    const uint32_t base28 = (uint32_t)kSmCls28 + 8u * u28, base143 = (uint32_t)kSmCls143 + 8u * u143;
    // k mod 143 slots: byte n of the step's word is taken from byte (n - m) mod 4, m = u143 mod 4,
    // so that lane l adds column (s + l - 8m) mod 32 there
    const uint32_t m = u143 & 3u;
    const uint32_t r143 = (lane - 8u * m) & 31u;
    uint32_t sel[4];
#pragma unroll
    for (uint32_t n = 0; n < 4; ++n) sel[n] = 0x4440u | ((n - m) & 3u);
#pragma unroll
    for (uint32_t s = 0; s < 32; ++s) {
      const uint32_t v28 = (tt[s & 7u] >> (8u * (s >> 3))) & 0xFFu;
      const uint32_t v143 = __byte_perm(tt[s & 7u], 0u, sel[s >> 3]);
      sm_add_n(cnt, base28 + ((s + lane) & 31u), v28, err);
      sm_add_n(cnt, base143 + ((s + r143) & 31u), v143, err);
    }
  }
}

// Mask of the bits of word w whose integers lie in [vlo, vhi); v0 = value of byte 4w, residue 0.
__device__ __forceinline__ uint32_t edge_mask(uint64_t v0, uint64_t vlo, uint64_t vhi) {
  uint32_t m = 0;
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j)
#pragma unroll
    for (uint32_t o = 0; o < 8; ++o) {
      uint64_t v = v0 + 30u * j + w30(o);
      if (v >= vlo && v < vhi) m |= 1u << (8u * j + o);
    }
  return m;
}

__device__ __forceinline__ uint32_t pre_mod(int g) {
  return g == 0 ? 1001u : (g == 1 ? 323u : (g == 2 ? 667u : 31u));
}
__device__ __forceinline__ uint32_t pre_off(int g) {
  return g == 0 ? 0u : (g == 1 ? 1001u : (g == 2 ? 1324u : 1991u));
}

#ifdef VOSS_PHASE_TIMING
// Instrumented build only: per-phase cycles summed over all CTAs (thread 0 of each CTA
// timestamps every phase boundary after a block barrier).
__device__ unsigned long long g_phase_cycles[16];
#define VOSS_PHASE(k)                                  \
  __syncthreads();                                     \
  if (threadIdx.x == 0) {                              \
    const long long now__ = clock64();                 \
    ph_acc[(k)] += (unsigned long long)(now__ - ph_t); \
    ph_t = now__;                                      \
  }
#else
#define VOSS_PHASE(k)
#endif

struct TileHdr {  // one tile's header (double-buffered: the next tile's is built during this one)
  unsigned long long ktile, vbase, vlo, vhi, seg_k;
  uint32_t nw, lt, np, ia, ib, iw, vb, cthr, k28, k143;
  uint32_t pre_base[kPreGroups];
  uint32_t interval, tile;
  uint32_t r0, r1;       // base primes lying in the tile (restore)
  uint32_t coop_ctr, b_ctr, w_ctr, c_ctr;  // work counters of the prime categories
  uint32_t w_items, w_item, w_lo[8], w_n[8];  // primes taken by class: items, primes per item, first and number per class
  unsigned long long gword;         // the tile's first word in the large-prime bitmap
  uint32_t first;
};

struct CtaState {  // what a CTA carries from tile to tile
  uint32_t cur_iv, since_flush, flush;
  uint32_t c_lt, c_ia, c_ib, c_iw;  // category bounds over the whole table for tile length c_lt
  unsigned long long count_total;
};

template <int BLOCK>
struct BlockScratch {
  int32_t warp_max[BLOCK / 32];
  int32_t warp_prefix[BLOCK / 32];
  int32_t block_max;
  uint32_t block_sum;
  uint32_t warp_sum[BLOCK / 32];
  unsigned long long warp_key[BLOCK / 32];
  bool redo;
};

// Exclusive sum-scan of `v` and max-scan of `m` over thread order in one pass, with the totals.
template <int BLOCK>
__device__ __forceinline__ void block_excl_sum_max(uint32_t v, int32_t m, BlockScratch<BLOCK>& S, uint32_t* sum_before,
                                                   uint32_t* sum, int32_t* max_before, int32_t* max_all) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t vi = v;
  int32_t mi = m;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t tv = __shfl_up_sync(0xFFFFFFFFu, vi, d);
    const int32_t tm = __shfl_up_sync(0xFFFFFFFFu, mi, d);
    if (lane >= d) {
      vi += tv;
      mi = max(mi, tm);
    }
  }
  if (lane == 31) {
    S.warp_sum[warp] = vi;
    S.warp_max[warp] = mi;
  }
  __syncthreads();
  if (warp == 0) {
    const uint32_t x = lane < BLOCK / 32 ? S.warp_sum[lane] : 0;
    uint32_t xi = x;
    int32_t yi = lane < BLOCK / 32 ? S.warp_max[lane] : -1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t tv = __shfl_up_sync(0xFFFFFFFFu, xi, d);
      const int32_t tm = __shfl_up_sync(0xFFFFFFFFu, yi, d);
      if (lane >= d) {
        xi += tv;
        yi = max(yi, tm);
      }
    }
    const int32_t ye = __shfl_up_sync(0xFFFFFFFFu, yi, 1);
    if (lane < BLOCK / 32) {
      S.warp_sum[lane] = xi - x;  // exclusive over the warps
      S.warp_prefix[lane] = lane == 0 ? -1 : ye;
    }
    if (lane == BLOCK / 32 - 1) {
      S.block_sum = xi;
      S.block_max = yi;
    }
  }
  __syncthreads();
  const int32_t me = __shfl_up_sync(0xFFFFFFFFu, mi, 1);
  *sum_before = vi - v + S.warp_sum[warp];
  *max_before = max(lane == 0 ? -1 : me, S.warp_prefix[warp]);
  *sum = S.block_sum;
  *max_all = S.block_max;
}

template <int BLOCK>
__device__ __forceinline__ uint32_t block_excl_sum(uint32_t v, BlockScratch<BLOCK>& S, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) S.warp_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t x = lane < BLOCK / 32 ? S.warp_sum[lane] : 0;
    uint32_t y = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t t = __shfl_up_sync(0xFFFFFFFFu, y, d);
      if (lane >= d) y += t;
    }
    if (lane < BLOCK / 32) S.warp_sum[lane] = y - x;  // exclusive prefix of warps
    if (lane == BLOCK / 32 - 1) S.warp_prefix[0] = (int32_t)y;
  }
  __syncthreads();
  uint32_t ex = incl - v + S.warp_sum[warp];
  *total = (uint32_t)S.warp_prefix[0];
  return ex;
}

// The largest key of the block, to thread 0.
template <int BLOCK>
__device__ __forceinline__ void block_max_key(unsigned long long key, BlockScratch<BLOCK>& S,
                                              unsigned long long* key_max) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    unsigned long long k2 = __shfl_down_sync(0xFFFFFFFFu, key, d);
    key = k2 > key ? k2 : key;
  }
  if (lane == 0) S.warp_key[warp] = key;
  __syncthreads();
  if (warp == 0) {
    unsigned long long k = lane < BLOCK / 32 ? S.warp_key[lane] : 0ull;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      unsigned long long k2 = __shfl_down_sync(0xFFFFFFFFu, k, d);
      k = k2 > k ? k2 : k;
    }
    if (lane == 0) *key_max = k;
  }
}

// Accumulator word of shared counter i, kNone for one that does not count (kSmSpare, distance 0).
// The class counters fold: shared class c of the (k mod 28) block is class c mod 28, of the
// (k mod 143) block class c mod 143.
__device__ __forceinline__ uint32_t acc_index(uint32_t i) {
  if (i < (uint32_t)kSmSpare) {
    const uint32_t d = i >> 3, o = i & 7u;
    if (d == 0) return kNone;
    const uint32_t g = 30u * ((o + d) >> 3) + w30((o + d) & 7u) - w30(o);
    return g < 2u * kModqBins ? (uint32_t)kAccModq + o * (uint32_t)kModqBins + (g >> 1) : (uint32_t)kAccHist + (g >> 1);
  }
  if (i < (uint32_t)kSmCls28) return kNone;
  if (i < (uint32_t)kSmCls143) {
    const uint32_t c = (i - (uint32_t)kSmCls28) >> 3;
    return (uint32_t)kAccCls28 + 8u * (c >= 28u ? c - 28u : c) + (i & 7u);
  }
  const uint32_t c = (i - (uint32_t)kSmCls143) >> 3;
  return (uint32_t)kAccCls143 + 8u * (c >= 143u ? c - 143u : c) + (i & 7u);
}

// Small primes' records (prime, remainder, residue class) take 13 + 13 + 3 bits of a word.
constexpr uint32_t kSmallPrimeEnd = 1u << 13;
// Lanes per prime of the progressions.  A warp's item is then 16 primes, and the longest item (640
// clears in a row for 32 primes above tile/80) no longer outlasts the others where few primes follow:
// [1, 10^9] 280 -> 252 us of tiles, one interval of 10^6 33 -> 28 us; 4 and 8 lanes cost long runs 1 and 2 %.
constexpr uint32_t kProgLanes = 2;

constexpr uint32_t kFlushEvery = 2048;  // tiles between counter flushes (u32 headroom)

// The header of tile t, built by one warp: the lanes compute the same scalars and share the
// table searches (count_le_warp); lane 0 writes the header.  t >= n_tiles marks the end.
__device__ __forceinline__ void tile_header(TileHdr& H, CtaState& St, const SieveArgs& a, uint32_t t,
                                            uint32_t ln) {
  {
    {
      const uint32_t ivx = t < a.n_tiles ? find_interval(a, t) : kNone;
      if (ln == 0) {
        H.tile = t;
        H.interval = ivx;
      }
      if (t >= a.n_tiles) return;
      const IntervalDev iv = a.iv[ivx];
      const uint32_t tl = t - iv.tile_begin;
      const uint64_t wofs = (uint64_t)tl * a.tile_words;
      const uint64_t nw64 = iv.n_words - wofs;
      const uint32_t nw = nw64 < a.tile_words ? (uint32_t)nw64 : a.tile_words;
      const uint64_t ktile = iv.k0 + 4ull * wofs;
      const uint64_t vbase = 30ull * ktile;
      const uint32_t lt = 4u * nw;
      uint64_t vend = vbase + 30ull * lt;
      if (vend > iv.hi) vend = iv.hi;
      // table searches, skipped where the answer is known: a tile past the table's last prime
      // needs every prime and holds none of them; the category bounds over the whole table
      // depend only on the tile length (count_lt over np primes = min(that, np))
      const uint64_t sq = isqrt_u64(vend - 1);
      uint32_t np = sq >= a.p_max ? a.n_primes : count_le_warp(a.primes, a.n_primes, sq, ln);
      if (a.gbm && np > a.scatter_first) np = a.scatter_first;  // the rest came from the pre-pass
      if (lt != St.c_lt) {
        // one record per thread of the block, and primes that fit a record (clear_small_prime)
        const uint32_t ia0 = count_lt_warp(a.primes, a.n_primes, (uint64_t)min(lt / a.coop_div, kSmallPrimeEnd), ln);
        const uint32_t ia = min(ia0, (uint32_t)blockDim.x);
        const uint32_t ib = count_lt_warp(a.primes, a.n_primes, a.p_large, ln);
        const uint32_t iw = count_lt_warp(a.primes, a.n_primes, ((uint64_t)lt * a.walk_sixteenths) >> 4, ln);
        __syncwarp();
        if (ln == 0) {
          St.c_ia = ia;
          St.c_ib = ib;
          St.c_iw = iw;
          St.c_lt = lt;
        }
        __syncwarp();
      }
      const uint32_t ia = min(St.c_ia, np);
      const uint32_t ib0 = min(St.c_ib, np);
      const uint32_t ib = ib0 < ia ? ia : ib0;
      // the by-class primes [iwb, ib): their lower end and the ascending list's upper end meet at a
      // multiple of kClsBlock, where the numbers of primes per class are tabulated; the upper end is
      // rounded up (a few primes beyond the tile's root or the pre-pass's first strike out
      // composites again)
      const uint32_t iwb = max(St.c_iw & ~(kClsBlock - 1u), (ia + kClsBlock - 1u) & ~(kClsBlock - 1u));
      const uint32_t iw = min(iwb, ib);
      uint32_t w_n = 0;
      if (ib > iwb && ln < 8u) {
        const uint32_t hb = min((ib + kClsBlock - 1u) / kClsBlock, a.n_cls_blocks);
        const uint32_t lo = a.cls_index[8u * (iwb / kClsBlock) + ln];
        w_n = a.cls_index[8u * hb + ln] - lo;
        H.w_lo[ln] = a.cls_first[ln] + lo;
        H.w_n[ln] = w_n;
      }
      // primes that a warp claims at a time: an item costs a claim and its class's constants (256
      // against 128 and 64: 18.40, 18.70 and 19.35 ms for the 10^11 integers below 10^12), but few
      // primes have to keep all warps busy
      const uint32_t w_max = __reduce_max_sync(0xFFFFFFFFu, w_n);
      const uint32_t w_item = w_max >= 4096u ? 256u : (w_max >= 1024u ? 128u : 32u);
      const uint32_t w_items = 8u * ((w_max + w_item - 1u) / w_item);
      // base primes that lie in the tile and may have been struck out as their own multiple: up to the
      // interval's root (the pre-pass), rounded up to a kClsBlock as above.  Below 2^24, where blocks
      // are in use, kClsBlock primes span less than 2^16; a context for 10^16 holds primes up to 10^8,
      // and restoring all of a tile's near 10^7 took 80 us.
      uint32_t r0 = a.n_primes, r1 = a.n_primes;
      const uint64_t root = vbase <= a.p_max ? isqrt_u64(iv.hi - 1) : 0;
      if (vbase <= a.p_max && vbase <= root + 65536u) {
        const uint32_t used = count_le_warp(a.primes, a.n_primes, root, ln) + kClsBlock;
        r0 = count_lt_warp(a.primes, a.n_primes, vbase, ln);
        r1 = min(count_lt_warp(a.primes, a.n_primes, vbase + 30ull * lt, ln), used);
      }
      if (ln == 0) {
        H.ktile = ktile;
        H.vbase = vbase;
        H.vlo = iv.lo;
        H.vhi = iv.hi;
        H.seg_k = iv.seg_k;
        H.nw = nw;
        H.lt = lt;
        H.np = np;
        H.gword = iv.gword + wofs;
        H.ia = ia;
        H.ib = ib;
        H.iw = iw;
        H.r0 = r0;
        H.r1 = r1;
        uint32_t vb = kNone;
        if (iv.seg_k) {
          uint64_t kb = (ktile / iv.seg_k + 1) * iv.seg_k;
          if (kb < ktile + lt) vb = (uint32_t)(30ull * (kb - ktile));
        }
        H.vb = vb;
        // large-gap candidates: g >= cthr, one tile-uniform threshold.  Reference rule
        // (voss_v7_live.cu:289-294): g > 100 and (g >= 500 or g / log(p) >= 10); no gap of the
        // tile below 10 log(vbase) - 3 can reach merit 10.  With large_min_gap: g >= large_min_gap.
        // (single-precision log: its error, a few units of 1e-6 relative at these sizes, is far
        // inside the margin of 3; the kept gaps are then decided by the double merit below)
        const float th = floorf(10.0f * __logf((float)(vbase > 7 ? vbase : 7))) - 3.0f;
        uint32_t gthr = th < 0.0f ? 0u : (uint32_t)th;
        gthr = gthr < 101u ? 101u : (gthr > 500u ? 500u : gthr);
        H.cthr = !a.want_large ? kNone : (a.large_min_gap ? a.large_min_gap : gthr);
        H.k28 = (uint32_t)(ktile % 28ull);
        H.k143 = (uint32_t)(ktile % 143ull);
        const uint64_t wt = ktile >> 2;
#pragma unroll
        for (int g = 0; g < kPreGroups; ++g) H.pre_base[g] = (uint32_t)(wt % pre_mod(g));
        H.coop_ctr = 0;
        H.b_ctr = 0;
        H.w_ctr = 0;
        H.w_items = w_items;
        H.w_item = w_item;
        H.c_ctr = 0;
        H.first = kNone;
      }
    }
  }
}

template <int BLOCK, bool EMIT>
__global__ void __launch_bounds__(BLOCK, (BLOCK == 512 ? 2 : 1))
sieve_tiles_kernel(SieveArgs a) {
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* bm = smem;
  uint32_t* pre = smem + a.tile_words + kSpareWords;
  uint32_t* cnt = pre + kPreWords;
  __shared__ TileHdr HH[2];  // this tile's header and the next one's
  __shared__ CtaState St;
  __shared__ BlockScratch<BLOCK> S;
  // Wheel tables in shared memory: lanes index them by their own prime's residue, which
  // would serialize in the constant cache.
  __shared__ __align__(8) uint8_t s_step[64];
  __shared__ int8_t s_rb[32];
  __shared__ uint32_t s_pos[32];  // bit b of a word -> integer offset 30 * (b / 8) + W30[b % 8]
  // extraction: first tile rank of each thread's chunk; sieve: the small primes' records
  __shared__ uint32_t s_rank[BLOCK];
  __shared__ int32_t s_before[EMIT ? 1 : BLOCK];  // last prime before each chunk (-1: none)
  __shared__ uint16_t s_mid[EMIT ? 1 : BLOCK];    // primes in the first C / 2 words of each chunk
  uint32_t* err = a.error;

  const int tid = threadIdx.x, lane = tid & 31;
  for (uint32_t i = tid; i < kPreWords; i += BLOCK) pre[i] = a.pretab[i];
  if (tid < 64) s_step[tid] = c_wheel_step.v[tid];
  if (tid < 32) s_rb[tid] = c_res_bit.v[tid];
  if (tid < 32) s_pos[tid] = 30u * ((uint32_t)tid >> 3) + w30((uint32_t)tid & 7u);
  if (!EMIT)
    for (uint32_t i = tid; i < (uint32_t)kSmCounters; i += BLOCK) cnt[i] = 0;
  if (tid == 0) {
    St.cur_iv = kNone;
    St.since_flush = 0;
    St.count_total = 0;
    St.c_lt = kNone;
  }
  __syncthreads();
  if (tid < 32) {  // the first tile: claim and header
    uint32_t t0 = 0;
    if (lane == 0) t0 = atomicAdd(a.tile_counter, 1u);
    tile_header(HH[0], St, a, __shfl_sync(0xFFFFFFFFu, t0, 0), (uint32_t)lane);
  }
  __syncthreads();
  uint32_t cur = 0;

  const uint32_t C = a.chunk_words;
#ifdef VOSS_PHASE_TIMING
  unsigned long long ph_acc[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  long long ph_t = clock64();
#endif

  for (;;) {
    TileHdr& H = HH[cur];  // built during the previous tile (or before the loop)
    // ---- flush ------------------------------------------------------------------------
    if (tid == 0) {
      const uint32_t ivx = H.tile < a.n_tiles ? H.interval : kNone;
      St.flush = (!EMIT && St.cur_iv != kNone &&
                  (ivx != St.cur_iv || St.since_flush >= kFlushEvery)) ? 1u : 0u;
    }
    __syncthreads();
    if (St.flush) {
      unsigned long long* acc = a.acc + (size_t)St.cur_iv * kAccStride;
      for (uint32_t i = tid; i < (uint32_t)kSmCounters; i += BLOCK) {
        uint32_t v = cnt[i];
        if (v) {
          const uint32_t k = acc_index(i);
          if (k != kNone) atomicAdd(acc + k, (unsigned long long)v);
          cnt[i] = 0;
        }
      }
      if (tid == 0) {
        atomicAdd(acc + kAccCount, St.count_total);
        St.count_total = 0;
        St.since_flush = 0;
      }
      __syncthreads();
    }
    if (H.tile >= a.n_tiles) break;
    if (tid == 0) St.cur_iv = H.interval;
    VOSS_PHASE(0)

    VOSS_PHASE(1)

    const uint32_t nw = H.nw, Lt = H.lt;
    // tiles below 2^53 reduce the prime offsets with one fma instead of the 64-bit Barrett product
    const bool fma_mod = H.vbase < (1ull << 53);
    const double ks = (double)H.ktile * 0x1p-64, vs = (double)H.vbase * 0x1p-64;

    // the small primes' records, a thread per prime: remainder of the tile's first byte, p, class
    if ((uint32_t)tid < H.ia) {
      const uint32_t p = a.primes[tid];
      const uint64_t m = a.magic[tid];
      const uint32_t r = fma_mod ? mod_by_magic_fma(H.ktile, ks, p, m) : mod_barrett(H.ktile, p, m);
      s_rank[tid] = r | p << 13 | (uint32_t)s_rb[p % 30u] << 26;
    }

    // ---- 1. fill ----------------------------------------------------------------------
    // Thread c < 1001 writes the words w = c (mod 1001): the mask of 7 * 11 * 13 is then the
    // thread's own constant, and the other tables' indices advance by fixed steps (three loads and
    // one store per word; 26k warp instructions less per tile than words tid + BLOCK k from four
    // tables with an edge test each).
    if (tid < 1001 || BLOCK < 1001) {
      const uint64_t vbase = H.vbase, vlo = H.vlo, vhi = H.vhi;
      const uint32_t* gbm = a.gbm ? a.gbm + H.gword : nullptr;
      // words [w_in, w_out) lie wholly inside [vlo, vhi) (v0 + 1 >= vlo and v0 + 120 <= vhi):
      // only the others need an edge mask
      const uint64_t lo_words = vlo <= vbase + 1 ? 0ull : (vlo - vbase + 118ull) / 120ull;
      const uint64_t hi_words = vhi < vbase + 120 ? 0ull : (vhi - vbase) / 120ull;
      const uint32_t w_in = (uint32_t)(lo_words < a.tile_words ? lo_words : a.tile_words);
      const uint32_t w_out = (uint32_t)(hi_words < nw ? hi_words : nw);
      for (uint32_t c = tid; c < 1001u; c += BLOCK) {
        uint32_t i0 = H.pre_base[0] + c, ix[kPreGroups];
        i0 -= i0 >= pre_mod(0) ? pre_mod(0) : 0u;
        const uint32_t m0 = pre[i0];
#pragma unroll
        for (int g = 1; g < kPreGroups; ++g) ix[g] = (H.pre_base[g] + c) % pre_mod(g);
        auto mask = [&] {
          const uint32_t m = m0 & pre[pre_off(1) + ix[1]] & pre[pre_off(2) + ix[2]] & pre[pre_off(3) + ix[3]];
#pragma unroll
          for (int g = 1; g < kPreGroups; ++g) {
            ix[g] += 1001u % pre_mod(g);
            ix[g] = min(ix[g], ix[g] - pre_mod(g));
          }
          return m;
        };
        uint32_t w = c;
        auto edge = [&](uint32_t end) {  // words that reach out of the interval
          for (; w < end; w += 1001u) {
            const uint32_t m = mask() & edge_mask(vbase + 120ull * w, vlo, vhi);
            bm[w] = gbm ? m & gbm[w] : m;
          }
        };
        edge(min(w_in, nw));
        if (gbm) {
          // the pre-pass's words, eight loads in flight per thread: one at a time they cost a tile 51
          // trips to L2 (4.7e9 integers near 10^15: 1172 -> 1095 us of tiles)
          for (; w + 7u * 1001u < w_out; w += 8u * 1001u) {
            uint32_t g[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) g[k] = __ldcg(gbm + w + 1001u * (uint32_t)k);
#pragma unroll
            for (int k = 0; k < 8; ++k) bm[w + 1001u * (uint32_t)k] = mask() & g[k];
          }
          for (; w < w_out; w += 1001u) bm[w] = mask() & __ldcg(gbm + w);
        } else {
#pragma unroll 4
          for (; w < w_out; w += 1001u) bm[w] = mask();
        }
        edge(nw);
      }
    }
    __syncthreads();
    VOSS_PHASE(2)

    // Warp 0 claims the next tile and builds its header now, while the other warps start on
    // this tile's small primes (claimed dynamically, so they take over warp 0's share): the
    // header's dependent loads no longer hold the whole CTA at a barrier between tiles.
    if (tid < 32) {
      uint32_t tn = 0;
      if (lane == 0) tn = atomicAdd(a.tile_counter, 1u);
      tile_header(HH[cur ^ 1u], St, a, __shfl_sync(0xFFFFFFFFu, tn, 0), (uint32_t)lane);
    }

    // ---- 2. sieve ----------------------------------------------------------------------
    {
      const uint64_t ktile = H.ktile;
      const uint32_t ia = H.ia, ib = H.ib, iw = H.iw, np = H.np;
      const TileBits T{bm, Lt + 4u * (uint32_t)lane, nw, err};
      // small primes: a warp per prime
      for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(&H.coop_ctr, 1u);
        i = __shfl_sync(0xFFFFFFFFu, i, 0);
        if (i >= ia) break;
        clear_small_prime(T, s_rank[i], s_step, (uint32_t)lane, Lt);
      }
      VOSS_PHASE(3)
      // medium primes
      if (a.b_mode == 0) {
        // kProgLanes lanes per prime, each some of its 8 residue progressions; warps claim 32 / kProgLanes
        // consecutive primes at a time
        constexpr uint32_t kPrimes = 32u / kProgLanes, kRes = 8u / kProgLanes;
        const uint32_t part = (uint32_t)lane / kPrimes;
        for (;;) {
          uint32_t base = 0;
          if (lane == 0) base = atomicAdd(&H.b_ctr, kPrimes);
          base = __shfl_sync(0xFFFFFFFFu, base, 0);
          if (base >= iw - ia) break;
          const uint32_t i = ia + base + (uint32_t)lane % kPrimes;
          if (i < iw) {
            const uint32_t p = a.primes[i];
            const uint64_t m = a.magic[i];
            const uint32_t r = fma_mod ? mod_by_magic_fma(ktile, ks, p, m) : mod_barrett(ktile, p, m);
            const uint32_t pa = p / 30u, bi = (uint32_t)s_rb[p - 30u * pa];
            const uint64_t st = *reinterpret_cast<const uint64_t*>(s_step + 8u * bi) >> (8u * kRes * part);
            const uint64_t wr = kW30Packed >> (8u * kRes * part);
#pragma unroll
            for (uint32_t o = 0; o < kRes; ++o) {
              const uint32_t e = (uint32_t)(st >> (8u * o)) & 0xFFu;
              const uint32_t delta = pa * ((uint32_t)(wr >> (8u * o)) & 0xFFu) + (e & 31u);
              clear_progression(T, delta >= r ? delta - r : delta + p - r, p, e >> 5, Lt);
            }
          }
        }
        // few hits per tile: a thread per prime of a class, 32 primes of one class at a time (item
        // i: class i mod 8, its (i / 8)-th item; the classes hold nearly equal numbers of primes)
        const double kd = (double)ktile;
        const uint32_t w_end = H.w_items, w_item = H.w_item;
        for (;;) {
          uint32_t it = 0;
          if (lane == 0) it = atomicAdd(&H.w_ctr, 1u);
          it = __shfl_sync(0xFFFFFFFFu, it, 0);
          if (it >= w_end) break;
          const uint32_t c = it & 7u, n = H.w_n[c];
          uint32_t k = w_item * (it >> 3);
          if (k >= n) continue;
          ClassStep C;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint2 e = c_cls_step.v[8u * c + j];
            C.corr[j] = e.x;
            C.bit[j] = e.y;
          }
          const uint32_t k_end = min(n, k + w_item);
          const uint32_t* pp = a.cls_primes + H.w_lo[c];
          const double* pi = a.cls_inv + H.w_lo[c];
          // idle lanes repeat the last prime; the next 32 primes are loaded ahead
          uint32_t i = min(k + (uint32_t)lane, n - 1u);
          uint32_t p = pp[i];
          double inv = pi[i];
          for (;;) {
            const uint32_t p_now = p;
            const double inv_now = inv;
            k += 32u;
            if (k < k_end) {
              i = min(k + (uint32_t)lane, n - 1u);
              p = pp[i];
              inv = pi[i];
            }
            const uint32_t r = mod_by_inv(ktile, kd, p_now, inv_now);
            const uint32_t pmin = __shfl_sync(0xFFFFFFFFu, p_now, 0);
            if (pmin >= Lt) clear_class_primes<true>(T, p_now, r, pmin, C, Lt);
            else clear_class_primes<false>(T, p_now, r, pmin, C, Lt);
            if (k >= k_end) break;
          }
        }
      } else {
        // a lane per (prime, residue): a warp takes 4 consecutive primes, lane = 8*prime + residue
        const uint32_t o = (uint32_t)lane & 7u;
        const uint32_t wo = w30(o);
        const uint32_t groups = (ib - ia + 3u) >> 2;
        const uint32_t warp = (uint32_t)tid >> 5;
        for (uint32_t g = warp; g < groups; g += BLOCK / 32) {
          const uint32_t i = ia + 4u * g + ((uint32_t)lane >> 3);
          if (i < ib) {
            const uint32_t p = a.primes[i];
            const uint32_t r = mod_barrett(ktile, p, a.magic[i]);
            const uint32_t pa = p / 30u, bi = (uint32_t)s_rb[p - 30u * pa];
            const uint32_t e = s_step[bi * 8u + o];
            const uint32_t delta = pa * wo + (e & 31u);
            clear_progression(T, delta >= r ? delta - r : delta + p - r, p, e >> 5, Lt);
          }
        }
      }
      VOSS_PHASE(4)
      // large primes: walk the multiples of p across the tile's span of integers
      const uint64_t vbase = H.vbase;
      const uint32_t span = 30u * Lt;
      for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&H.c_ctr, 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= np - ib) break;
        const uint32_t i = ib + base + (uint32_t)lane;
        if (i < np) {
          const uint32_t p = a.primes[i];
          const uint64_t m = a.magic[i];
          const uint32_t r = fma_mod && p < (1u << 30) ? mod_by_magic_fma(vbase, vs, p, m) : mod_barrett(vbase, p, m);
          uint32_t d = r ? p - r : 0u;
          for (; d < span; d += p) {
            const uint32_t q = d / 30u;
            const int b = s_rb[d - 30u * q];
            if (b >= 0) T.clear(q & ~3u, bit_mask(q, (uint32_t)b));
          }
        }
      }
    }
    __syncthreads();
    VOSS_PHASE(5)

    // ---- 3. restore primes lying in the tile ---------------------------------------------
    if (H.vbase < 32 || H.r0 < H.r1) {
      const uint64_t vbase = H.vbase, vlo = H.vlo, vhi = H.vhi, vend = vbase + 30ull * Lt;
      if (vbase < 32 && tid < 8) {
        const uint32_t sp[8] = {7, 11, 13, 17, 19, 23, 29, 31};
        const uint64_t p = sp[tid];
        if (p >= vlo && p < vhi && p >= vbase && p < vend) {
          const uint32_t off = (uint32_t)(p - vbase), k = off / 30u;
          atomicOr(bm + (k >> 2), 1u << (((k & 3u) << 3) | (uint32_t)s_rb[off - 30u * k]));
        }
      }
      for (uint32_t i = H.r0 + tid; i < H.r1; i += BLOCK) {
        const uint64_t p = a.primes[i];
        if (p >= vlo && p < vhi && p >= vbase && p < vend) {
          const uint32_t off = (uint32_t)(p - vbase), k = off / 30u;
          if ((k >> 2) < nw)
            atomicOr(bm + (k >> 2), 1u << (((k & 3u) << 3) | (uint32_t)s_rb[off - 30u * k]));
        }
      }
      __syncthreads();
    }
    VOSS_PHASE(6)

    // ---- 4. extract -----------------------------------------------------------------------
    const uint32_t c0 = (uint32_t)tid * C;
    const uint32_t cend = c0 < nw ? (c0 + C < nw ? c0 + C : nw) : c0;

    if (EMIT) {
      uint32_t pc = 0;
      for (uint32_t w = c0; w < cend; ++w) pc += __popc(bm[w]);
      uint32_t total;
      uint32_t rank = block_excl_sum<BLOCK>(pc, S, &total);
      const unsigned long long base = a.tile_offset[H.tile];
      const uint64_t vbase = H.vbase;
      for (uint32_t w = c0; w < cend; ++w) {
        uint32_t x = bm[w];
        while (x) {
          const uint32_t b = (uint32_t)__ffs(x) - 1u;
          x &= x - 1u;
          const unsigned long long idx = base + rank;
          if (idx < a.out_cap) a.out[idx] = vbase + 120ull * w + 30u * (b >> 3) + w30(b & 7u);
          ++rank;
        }
      }
      __syncthreads();
    } else {
      class_counts_by_word<BLOCK>(bm, nw, H.k28, H.k143, cnt, (uint32_t)lane, err);
      // pass 1: the primes of my chunk and its last prime
      uint32_t pc = 0;
      int32_t my_last = -1;
      const uint32_t cmid = c0 + (C >> 1) < cend ? c0 + (C >> 1) : cend;
#pragma unroll 4
      for (uint32_t w = c0; w < cmid; ++w) pc += (uint32_t)__popc(bm[w]);
      const uint32_t pc_half = pc;
#pragma unroll 4
      for (uint32_t w = cmid; w < cend; ++w) pc += (uint32_t)__popc(bm[w]);
      for (uint32_t w = cend; pc && w > c0;) {  // the chunk's last prime: its last non-zero word
        const uint32_t x = bm[--w];
        if (x) {
          my_last = (int32_t)(32u * w + 31u - (uint32_t)__clz(x));
          break;
        }
      }
      uint32_t tile_cnt, rank0;
      int32_t tile_last, before;
      block_excl_sum_max<BLOCK>(pc, my_last, S, &rank0, &tile_cnt, &before, &tile_last);
      s_rank[tid] = rank0;
      s_mid[tid] = (uint16_t)pc_half;
      s_before[tid] = before;
      __syncthreads();
      VOSS_PHASE(7)

      // pass 2: every thread walks the same number of the tile's primes in order (ranks
      // [ra, rb) of tile_cnt), so that the lanes of a warp run the same trip count.  The start
      // is the prime of rank ra: the chunk holding it is the last one whose first rank is <= ra.
      const uint32_t ra = (uint32_t)(((unsigned long long)tile_cnt * (uint32_t)tid) / BLOCK);
      const uint32_t rb = (uint32_t)(((unsigned long long)tile_cnt * ((uint32_t)tid + 1u)) / BLOCK);
      const uint32_t n_mine = rb - ra;
      uint32_t w = 0, x = 0;
      int32_t prev = -1;
      if (n_mine) {
        uint32_t lo = 0, hi = BLOCK;  // s_rank[lo] <= ra
        while (hi - lo > 1u) {
          const uint32_t mid = (lo + hi) >> 1;
          if (s_rank[mid] <= ra) lo = mid; else hi = mid;
        }
        uint32_t k = ra - s_rank[lo];
        w = lo * C;
        const uint32_t kh = s_mid[lo];
        if (k >= kh) {  // the start lies in the chunk's second half
          k -= kh;
          w += C >> 1;
        }
        x = bm[w];
        for (;;) {  // the word holding the start: it lies in chunk lo
          const uint32_t c = (uint32_t)__popc(x);
          if (k < c) break;
          k -= c;
          x = bm[++w];
        }
        if (k) {  // the primes of that word before mine: the last of them is my predecessor
          for (; k > 1u; --k) x &= x - 1u;
          prev = (int32_t)(32u * w + (uint32_t)__ffs(x) - 1u);
          x &= x - 1u;
        } else {  // mine is the word's first prime: the predecessor is in an earlier word
          prev = s_before[lo];
          for (uint32_t ww = w; ww > lo * C;) {
            const uint32_t y = bm[--ww];
            if (y) {
              prev = (int32_t)(32u * ww + 31u - (uint32_t)__clz(y));
              break;
            }
          }
        }
      }
      // The walk works in bitmap bits (bit 8k + o of the tile = integer 30k + W30[o]): one counter
      // per (distance d, residue of the lower prime), no conversion to integers.  Only gaps of at
      // least t_far bits are looked at closer (far_gap): t_far is such that every large-gap
      // candidate is one (a gap of g holds at least 8g/30 - 0.87 bits), and about thirty others of
      // the tile, so that the longest gap is found among them.  If it is not clear that it was (a
      // gap below t_far bits is below 3.75 t_far), the tile's gaps are gone through again.
      // Bound by issue slots: 294k warp instructions per tile of 218,000 primes (near 10^12) with positions
      // as integers, a branch per reload and the longest gap tracked per prime; 205k with bit distances and
      // one vote; the step to the next word as one predicated sequence on its address took another 5 %
      // off the whole kernel (17.7 -> 16.9 ms for the 10^11 integers below 10^12).
      const uint32_t cthr = H.cthr;
      uint32_t t_far;
      {
        const float bits = 32.0f * (float)nw / (float)(tile_cnt | 1u);
        const float t = bits * __logf((float)(tile_cnt | 1u) * (1.0f / 32.0f));
        t_far = t < 1.0f ? 1u : (t > (float)kGapBits ? kGapBits : (uint32_t)t);
        if (cthr < 2u * kGapBits * 15u / 8u) t_far = min(t_far, max(1u, 8u * cthr / 30u));
      }
      uint32_t mg = 0, mlo = 0;
      // bits are counted from shared-memory address 0, so a word's address gives its first bit
      const uint32_t sb = (uint32_t)__cvta_generic_to_shared(bm), bit0 = 8u * sb;
      auto value = [&](uint32_t bit) { return 120u * ((bit - bit0) >> 5) + s_pos[(bit - bit0) & 31u]; };
      auto far_gap = [&](uint32_t lo_bit, uint32_t hi_bit, bool crossing) {
        const uint32_t pv = value(lo_bit), pos = value(hi_bit), g = pos - pv;
        if (crossing || hi_bit - lo_bit >= kGapBits) {  // not counted in shared memory
          unsigned long long* acc = a.acc + (size_t)H.interval * kAccStride;
          if (g < 2u * kHistBins) {
            atomicAdd(acc + kAccHist + (g >> 1), 1ull);
          } else {
            atomicAdd(acc + kAccHistOver, 1ull);
            const uint32_t slot = atomicAdd(a.over_count, 1u);
            if (slot < a.over_cap) a.over[slot] = OverflowGap{H.interval, g};
            else atomicOr(err, kErrOverflowList);
          }
        }
        mlo = g > mg ? pv : mlo;
        mg = g > mg ? g : mg;
        if (g >= cthr && !crossing) {
          const uint64_t v0 = H.vbase + pv;
          const double merit_d = (double)g / log((double)v0);
          if (a.large_min_gap || g >= 500u || merit_d >= 10.0) {
            const uint32_t slot = atomicAdd(a.large_count, 1u);
            if (slot < a.large_cap) {
              a.large[slot] = LargeGapDev{H.vbase + pos, (int32_t)g, (float)merit_d};
              a.large_iv[slot] = H.interval;
            }
          }
        }
      };
      uint32_t left = n_mine;
      uint32_t wp = sb + 4u * w;  // address of the word that x comes from
      if (n_mine)
        while (x == 0u) next_word_if_spent(x, wp);  // the tile holds this thread's primes: wp stays inside it
      if (prev < 0 && n_mine) {
        // the tile's first prime: no predecessor in the tile (exactly one thread)
        prev = (int32_t)(8u * (wp - sb) + (uint32_t)__ffs(x) - 1u);
        x &= x - 1u;
        H.first = value(bit0 + (uint32_t)prev);
        --left;
        if (left)
          while (x == 0u) next_word_if_spent(x, wp);
      }
      uint32_t pv = bit0 + (uint32_t)prev;
      const uint32_t vb = H.vb == kNone ? kNone : bit0 + 8u * (H.vb / 30u);  // the boundary's first bit
      // Instantiated twice: in a tile without a segment boundary (nearly all of them) the crossing
      // test drops out of the loop.
      auto walk = [&](auto cross_tag) {
        constexpr bool kCross = decltype(cross_tag)::value;
        // All but the last prime, the warp's lanes side by side: the next word is a predicated load,
        // and one vote covers what is rare, a far gap or a word without primes (a branch of its own
        // for the reload diverges at nearly every prime).
        const uint32_t common = __reduce_min_sync(0xFFFFFFFFu, left);
#pragma unroll 4
        for (uint32_t it = 1; it < common; ++it) {
          const uint32_t bit = 8u * wp + (uint32_t)__ffs(x) - 1u;
          x &= x - 1u;
          next_word_if_spent(x, wp);
          const uint32_t d = bit - pv;
          const bool crossing = kCross && (pv < vb) && (bit >= vb);
          const uint32_t slot = min(8u * d + (pv & 7u), (uint32_t)kSmSpare);
          sm_add(cnt, crossing ? (uint32_t)kSmSpare : slot, err);
          const bool far = d >= t_far || crossing;
          if (__any_sync(0xFFFFFFFFu, far || x == 0u)) {
            if (far) far_gap(pv, bit, crossing);
            while (x == 0u) next_word_if_spent(x, wp);  // this lane has primes left
          }
          pv = bit;
        }
        left -= common ? common - 1u : 0u;
        for (; left; --left) {
          while (x == 0u) next_word_if_spent(x, wp);
          const uint32_t bit = 8u * wp + (uint32_t)__ffs(x) - 1u;
          x &= x - 1u;
          const uint32_t d = bit - pv;
          const bool crossing = kCross && (pv < vb) && (bit >= vb);
          const uint32_t slot = min(8u * d + (pv & 7u), (uint32_t)kSmSpare);
          sm_add(cnt, crossing ? (uint32_t)kSmSpare : slot, err);
          if (d >= t_far || crossing) far_gap(pv, bit, crossing);
          pv = bit;
        }
      };
      if (vb == kNone) walk(std::false_type{});
      else walk(std::true_type{});
      auto gap_key = [&] {
        return mg ? (((unsigned long long)mg << 32) | (unsigned long long)(0xFFFFFFFFu - mlo)) : 0ull;
      };
      auto store_partial = [&](unsigned long long key) {
        TilePartial P;
        P.first = tile_cnt ? H.first : kNone;
        P.last = tile_cnt ? value(bit0 + (uint32_t)tile_last) : kNone;
        P.count = tile_cnt;
        P.max_gap = (uint32_t)(key >> 32);
        P.max_lo = key ? 0xFFFFFFFFu - (uint32_t)(key & 0xFFFFFFFFull) : 0u;
        P.bgap = 0;
        P.bgap_lo = 0;
        a.partials[H.tile] = P;
      };
      unsigned long long tile_key;
      __syncthreads();  // H.first visible, scratch reuse
      VOSS_PHASE(8)
      block_max_key<BLOCK>(gap_key(), S, &tile_key);
      if (tid == 0) {
        store_partial(tile_key);
        S.redo = tile_cnt >= 2u && 4u * (uint32_t)(tile_key >> 32) < 15u * t_far;
        St.count_total += tile_cnt;
        St.since_flush++;
      }
      __syncthreads();
      if (S.redo) {  // the longest gap may be a short one: every chunk's gaps in order
        mg = mlo = 0;
        int32_t pb = s_before[tid];
        for (uint32_t ww = c0; ww < cend; ++ww) {
          for (uint32_t y = bm[ww]; y; y &= y - 1u) {
            const uint32_t bit = 32u * ww + (uint32_t)__ffs(y) - 1u;
            if (pb >= 0) {
              const uint32_t lo_v = value(bit0 + (uint32_t)pb), g = value(bit0 + bit) - lo_v;
              mlo = g > mg ? lo_v : mlo;
              mg = g > mg ? g : mg;
            }
            pb = (int32_t)bit;
          }
        }
        block_max_key<BLOCK>(gap_key(), S, &tile_key);
        if (tid == 0) store_partial(tile_key);
      }
    }
    cur ^= 1u;
    __syncthreads();
    VOSS_PHASE(9)
  }
#ifdef VOSS_PHASE_TIMING
  if (threadIdx.x == 0)
    for (int k = 0; k < 10; ++k) atomicAdd(&g_phase_cycles[k], ph_acc[k]);
#endif
}

// The gap between the last prime of the previous non-empty tile and tile t's first prime (P, not
// empty): counted, and kept in *gap / *gap_lo (0: none).
__device__ __forceinline__ void tile_seam(const SieveArgs& a, const IntervalDev& iv, uint32_t ivx, uint32_t t,
                                          const TilePartial& P, uint32_t* gap, uint64_t* gap_lo) {
  *gap = 0;
  *gap_lo = 0;
  uint32_t tp = t;
  bool found = false;
  while (tp > iv.tile_begin) {
    --tp;
    if (a.partials[tp].count) {
      found = true;
      break;
    }
  }
  if (!found) return;
  const uint64_t kt = iv.k0 + 4ull * a.tile_words * (t - iv.tile_begin);
  const uint64_t kp = iv.k0 + 4ull * a.tile_words * (tp - iv.tile_begin);
  const uint64_t hi_p = 30ull * kt + P.first;
  const uint64_t lo_p = 30ull * kp + a.partials[tp].last;
  const uint64_t g = hi_p - lo_p;
  const bool crossing = iv.seg_k && ((lo_p / 30ull) / iv.seg_k != (hi_p / 30ull) / iv.seg_k);
  unsigned long long* acc = a.acc + (size_t)ivx * kAccStride;
  if (g < 100 && !crossing) {
    const uint32_t o_prev = (uint32_t)c_res_bit.v[lo_p % 30ull];
    atomicAdd(acc + kAccModq + o_prev * kModqBins + (g >> 1), 1ull);
  } else if (g < 2ull * kHistBins) {
    atomicAdd(acc + kAccHist + (g >> 1), 1ull);
  } else {
    atomicAdd(acc + kAccHistOver, 1ull);
    const uint32_t slot = atomicAdd(a.over_count, 1u);
    if (slot < a.over_cap) a.over[slot] = OverflowGap{ivx, (uint32_t)(g > 0xFFFFFFFFull ? 0xFFFFFFFFull : g)};
    else atomicOr(a.error, kErrOverflowList);
  }
  *gap = (uint32_t)(g > 0xFFFFFFFFull ? 0xFFFFFFFFull : g);
  *gap_lo = lo_p;
  const bool cand = a.large_min_gap ? (g >= a.large_min_gap) : (g > 100);
  if (a.want_large && cand && !crossing) {
    const double merit_d = (double)g / log((double)lo_p);
    if (a.large_min_gap || g >= 500 || merit_d >= 10.0) {
      const uint32_t slot = atomicAdd(a.large_count, 1u);
      if (slot < a.large_cap) {
        a.large[slot] = LargeGapDev{hi_p, (int32_t)g, (float)merit_d};
        a.large_iv[slot] = ivx;
      }
    }
  }
}

// The seams of a launch with many tiles per interval, a thread per tile (kept in the partials).
__global__ void stitch_kernel(SieveArgs a) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_tiles) return;
  const TilePartial P = a.partials[t];
  if (P.count == 0) return;
  const uint32_t ivx = find_interval(a, t);
  const IntervalDev iv = a.iv[ivx];
  uint32_t gap;
  uint64_t gap_lo;
  tile_seam(a, iv, ivx, t, P, &gap, &gap_lo);
  a.partials[t].bgap = gap;
  a.partials[t].bgap_lo = gap_lo;
}

// One block per interval, after its tiles: the seams between them (unless stitch_kernel ran), first
// and last prime, the first maximal gap; with `stats`, the accumulators folded into
// voss_interval_stats, so that only the result crosses to the host (lo, hi and the primes 2, 3, 5
// are filled in there).  One launch instead of three of 2 to 5 us each, which a launch of a few
// tiles notices.
constexpr int kTailBlock = 256;

__global__ void __launch_bounds__(kTailBlock) tail_kernel(SieveArgs a, bool stitched, IntervalOut* out,
                                                          voss_interval_stats* stats, const uint32_t* out_index) {
  const uint32_t ivx = blockIdx.x;
  const IntervalDev iv = a.iv[ivx];
  __shared__ uint32_t s_first, s_last;
  __shared__ unsigned long long s_gap[kTailBlock / 32], s_lo[kTailBlock / 32];
  if (threadIdx.x == 0) {
    s_first = kNone;
    s_last = 0;
  }
  __syncthreads();
  uint32_t my_first = kNone, my_last = 0;
  unsigned long long my_gap = 0, my_lo = ~0ull;
  auto longer = [&](unsigned long long g, unsigned long long lo) {  // ties: the smaller lower prime
    if (g > my_gap || (g == my_gap && lo < my_lo)) {
      my_gap = g;
      my_lo = lo;
    }
  };
  for (uint32_t i = threadIdx.x; i < iv.n_tiles; i += kTailBlock) {
    const TilePartial P = a.partials[iv.tile_begin + i];
    if (!P.count) continue;
    my_first = min(my_first, i);
    my_last = max(my_last, i + 1);
    uint32_t bgap = P.bgap;
    uint64_t bgap_lo = P.bgap_lo;
    if (!stitched) tile_seam(a, iv, ivx, iv.tile_begin + i, P, &bgap, &bgap_lo);
    if (P.max_gap) longer(P.max_gap, 30ull * (iv.k0 + 4ull * a.tile_words * i) + P.max_lo);
    if (bgap) longer(bgap, bgap_lo);
  }
  atomicMin(&s_first, my_first);
  atomicMax(&s_last, my_last);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const unsigned long long g = __shfl_down_sync(0xFFFFFFFFu, my_gap, d);
    const unsigned long long lo = __shfl_down_sync(0xFFFFFFFFu, my_lo, d);
    longer(g, lo);
  }
  if ((threadIdx.x & 31) == 0) {
    s_gap[threadIdx.x >> 5] = my_gap;
    s_lo[threadIdx.x >> 5] = my_lo;
  }
  __threadfence();  // the seams of the block are in the accumulators
  __syncthreads();
  voss_interval_stats* s = stats ? stats + (out_index ? out_index[ivx] : ivx) : nullptr;
  const unsigned long long* A = a.acc + (size_t)ivx * kAccStride;
  if (threadIdx.x == 0) {
    for (int w = 1; w < kTailBlock / 32; ++w) longer(s_gap[w], s_lo[w]);
    IntervalOut o;
    o.first = o.last = 0;
    if (s_first != kNone) {
      const TilePartial F = a.partials[iv.tile_begin + s_first];
      const TilePartial L = a.partials[iv.tile_begin + s_last - 1];
      o.first = 30ull * (iv.k0 + 4ull * a.tile_words * s_first) + F.first;
      o.last = 30ull * (iv.k0 + 4ull * a.tile_words * (s_last - 1)) + L.last;
    }
    o.max_gap = my_gap;
    o.max_gap_lo = my_gap ? my_lo : 0;
    out[ivx] = o;
    if (s) {
      s->lo = 0;
      s->hi = 0;
      s->prime_count = __ldcg(A + kAccCount);
      s->first_prime = o.first;
      s->last_prime = o.last;
      s->max_gap = o.max_gap;
      s->max_gap_lo = o.max_gap_lo;
      s->gap_overflow = __ldcg(A + kAccHistOver);
    }
  }
  if (!s) return;
  for (uint32_t b = threadIdx.x; b < (uint32_t)VOSS_IHIST; b += kTailBlock) {
    unsigned long long v = 0;
    if (b > 0) {
      v = __ldcg(A + kAccHist + b);
      if (b < (uint32_t)kModqBins)
        for (uint32_t o = 0; o < 8; ++o) v += __ldcg(A + kAccModq + o * kModqBins + b);
    }
    s->gap_hist[b] = v;
  }
}

// Zeroes the launch's counters and accumulators and fills its large-prime bitmap with ones in one
// launch (a memset of each takes about as long).
__global__ void init_kernel(uint4* zero, size_t n_zero, uint32_t* ones, size_t n_ones) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (size_t i = first; i < n_zero; i += stride) zero[i] = make_uint4(0, 0, 0, 0);
  uint4* ones4 = reinterpret_cast<uint4*>(ones);
  for (size_t i = first; i < n_ones / 4; i += stride) ones4[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (size_t i = (n_ones & ~(size_t)3) + first; i < n_ones; i += stride) ones[i] = ~0u;
}

int launch_init(void* zero, size_t zero_bytes, uint32_t* ones, size_t n_ones, int sm_count, void* stream) {
  const size_t n_zero = zero_bytes / sizeof(uint4);
  const size_t want = (std::max(n_zero, n_ones / 4) + 255) / 256 + 1;
  const int grid = (int)std::min<size_t>(want, (size_t)sm_count * 16);
  init_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((uint4*)zero, n_zero, ones, n_ones);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Large-prime pre-pass (bucket-free): each lane takes primes p >= p_large in turn and, for every
// interval of the launch that p can reach (intervals sorted by isqrt(hi - 1), descending, staged in
// shared memory), finds p's first multiple in it; p's multiples across the interval are cleared in the
// launch's large-prime bitmap with global atomics.  The prime table is read once
// per launch instead of once per tile, which is what bounds high intervals (at 1e18 the table
// is 610 MB).  The tile kernel ANDs this bitmap into its fill and skips these primes.
constexpr int kScatterChunk = 512;  // 24 KB of interval descriptors per block
constexpr int kScatterBlock = 512;
constexpr uint32_t kScatterQueue = 96;  // at most 31 waiting + 2 * 32 arriving

// A (prime, interval) pair with a multiple inside: d = the first multiple's offset from the
// interval's base.  The pairs that have one wait in the warp's queue and are walked 32 at a time, a
// lane each: among 32 primes of one interval a few to all have one, and each has another number.
// Over the 4096-interval batch (2.7e9 pairs, 9.5e8 clears) the pre-pass takes 7.8 ms against 8.9 with
// every pair walked where it is found: 0.21, 0.68, 1.53 and 5.9 ms for the intervals of 10^4..10^5,
// ..10^6, ..10^7 and ..10^8 against 0.33, 1.17, 2.33 and 6.0.  The long ones are bound by the atomics
// (3.5 ms without them), whose 32 lanes hit 32 sectors.
struct ScatterQueue {
  uint32_t d[kScatterQueue], p[kScatterQueue], s[kScatterQueue];
};

__device__ __forceinline__ void scatter_walk(const IntervalScatter& I, uint32_t d, uint32_t p, const int8_t* s_rb,
                                             const uint8_t* s_wstart, const uint2* s_wstep, uint32_t* __restrict__ gbm) {
  // wheel walk over the multiples p*m with gcd(m, 30) = 1 (vbase is a multiple of 30)
  const uint32_t pa = p / 30u, bi = (uint32_t)s_rb[p - 30u * pa];
  const uint32_t st = s_wstart[bi * 30u + (d - 30u * (d / 30u))];
  const uint64_t off = (uint64_t)d + (uint64_t)(st & 7u) * p;
  if (off >= I.span32) return;
  uint32_t byte = (uint32_t)off / 30u, w = st >> 3;
  const uint32_t lt = I.lt32;
  const uint2* row = s_wstep + bi * 8u;
  uint32_t* g = gbm + I.gword;
  do {
    const uint2 e = row[w];
    atomicAnd(g + (byte >> 2), __funnelshift_l(e.x, e.x, byte << 3));
    byte += pa * (e.y & 0xFFFFu) + (e.y >> 16);
    w = (w + 1u) & 7u;
  } while (byte < lt);
}

__global__ void __launch_bounds__(kScatterBlock) scatter_large_kernel(const uint32_t* __restrict__ primes, uint32_t j0,
                                                                      uint32_t j1,
                                                                      const IntervalScatter* __restrict__ iv,
                                                                      uint32_t n_iv, uint32_t* __restrict__ gbm) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  __shared__ IntervalScatter s_iv[kScatterChunk];
  __shared__ ScatterQueue s_q[kScatterBlock / 32];
  __shared__ int8_t s_rb[32];
  __shared__ uint8_t s_wstart[240];
  __shared__ uint2 s_wstep[64];
  if (threadIdx.x < 32) s_rb[threadIdx.x] = c_res_bit.v[threadIdx.x];
  if (threadIdx.x < 240) s_wstart[threadIdx.x] = c_walk_start.v[threadIdx.x];
  if (threadIdx.x < 64) s_wstep[threadIdx.x] = c_walk_step.v[threadIdx.x];
  for (uint32_t i = threadIdx.x; i < n_iv; i += blockDim.x) s_iv[i] = iv[i];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  ScatterQueue& Q = s_q[threadIdx.x >> 5];
  uint32_t nq = 0;
  auto add = [&](bool hit, uint32_t d, uint32_t p, uint32_t s) {
    const unsigned m = __ballot_sync(kFull, hit);
    if (hit) {
      const uint32_t at = nq + (uint32_t)__popc(m & ((1u << lane) - 1u));
      Q.d[at] = d;
      Q.p[at] = p;
      Q.s[at] = s;
    }
    nq += (uint32_t)__popc(m);
  };
  auto walk = [&](uint32_t n) {  // the last n <= 32 entries
    __syncwarp();
    nq -= n;
    if (lane < n) scatter_walk(s_iv[Q.s[nq + lane]], Q.d[nq + lane], Q.p[nq + lane], s_rb, s_wstart, s_wstep, gbm);
    __syncwarp();
  };
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t jb = j0 + blockIdx.x * blockDim.x + (threadIdx.x & ~31u); jb < j1; jb += stride) {
    const uint32_t j = min(jb + lane, j1 - 1u);
    const uint32_t p = primes[j];  // >= 2^13 (choose_shape); with the smallest tile that can be set >= 2^11
    const double inv = __drcp_rn((double)p);
    // intervals are sorted by sqrt_hi, descending: p reaches the first n_reach of them
    uint32_t lo = 0, hi = jb + lane < j1 ? n_iv : 0;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (s_iv[mid].sqrt_hi >= p) lo = mid + 1; else hi = mid;
    }
    const uint32_t n_reach = lo, reach_w = __reduce_max_sync(kFull, n_reach);
    if (__all_sync(kFull, p < (1u << 30))) {
      // The first multiple's offset d = q p - vbase with q = vbase / p rounded to an integer (adding
      // 2^52 in the same rounding leaves it in the low mantissa bits: q < 2^51 for vbase < 2^62): vd and
      // inv are off by a relative 2^-53 each, so |d| < 0.63 p for p >= 2^13 and below p for p >= 2^11.
      // The low 32 bits hold it, and a negative one needs one p more.
      auto first = [&](const uint4& h) {  // h: one 16-byte load per pair (vbase_d, vbase_lo, span32)
        const double vd = __hiloint2double((int)h.y, (int)h.x);
        const uint32_t d = (uint32_t)__double2loint(__fma_rn(vd, inv, 4503599627370496.0)) * p - h.z;
        return min(d, d + p);
      };
      for (uint32_t s = 0; s < reach_w; s += 2) {
        const uint4 h0 = *reinterpret_cast<const uint4*>(&s_iv[s]);
        const uint4 h1 = *reinterpret_cast<const uint4*>(&s_iv[min(s + 1u, reach_w - 1u)]);
        const uint32_t d0 = first(h0), d1 = first(h1);
        const bool hit0 = d0 < h0.w && s < n_reach, hit1 = d1 < h1.w && s + 1u < n_reach;
        if (!__any_sync(kFull, hit0 || hit1)) continue;
        add(hit0, d0, p, s);
        add(hit1, d1, p, s + 1u);
        while (nq >= 32u) walk(32u);
      }
    } else {  // primes of 2^30 and more (hi above 2^60): 64-bit remainders
      for (uint32_t s = 0; s < reach_w; ++s) {
        const IntervalScatter& I = s_iv[s];
        const double qd = __fma_rn(I.vbase_d, inv, 4503599627370496.0);
        const unsigned long long q = (unsigned long long)(__double_as_longlong(qd) - 0x4330000000000000ll);
        int64_t rr = (int64_t)(I.vbase - q * (uint64_t)p);
        rr += rr < 0 ? (int64_t)p : 0;
        rr -= rr >= (int64_t)p ? (int64_t)p : 0;
        const uint32_t d = rr ? p - (uint32_t)rr : 0u;
        add(d < I.span32 && s < n_reach, d, p, s);
        while (nq >= 32u) walk(32u);
      }
    }
  }
  if (nq) walk(nq);
}

int launch_scatter_large(const uint32_t* primes, uint32_t j0, uint32_t j1, const IntervalScatter* iv, uint32_t n_iv,
                         uint32_t* gbm, int sm_count, void* stream, uint32_t* kernels) {
  if (j1 <= j0 || n_iv == 0) return 0;
  const uint64_t want = ((uint64_t)(j1 - j0) + kScatterBlock - 1) / kScatterBlock;
  const int grid = (int)(want < (uint64_t)sm_count * 4 ? want : (uint64_t)sm_count * 4);
  for (uint32_t off = 0; off < n_iv; off += kScatterChunk) {
    const uint32_t n = n_iv - off < (uint32_t)kScatterChunk ? n_iv - off : (uint32_t)kScatterChunk;
    scatter_large_kernel<<<grid, kScatterBlock, 0, (cudaStream_t)stream>>>(primes, j0, j1, iv + off, n, gbm);
    ++*kernels;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// ---- shared-memory RMW probe ------------------------------------------------------------
constexpr int kProbeWords = 8192;
constexpr int kProbeIters = 4096;

__global__ void __launch_bounds__(1024) smem_rmw_probe_kernel(uint32_t* sink) {
  __shared__ uint32_t s[kProbeWords];
  for (int i = threadIdx.x; i < kProbeWords; i += blockDim.x) s[i] = 0xFFFFFFFFu;
  __syncthreads();
  uint32_t idx = threadIdx.x;
#pragma unroll 8
  for (int it = 0; it < kProbeIters; ++it) {
    atomicAnd(&s[idx & (kProbeWords - 1)], ~(1u << (it & 31)));
    idx += 1024u;
  }
  __syncthreads();
  if (threadIdx.x == 0) sink[blockIdx.x] = s[blockIdx.x & (kProbeWords - 1)];
}

// ---- host side ------------------------------------------------------------------------------
#ifdef VOSS_PHASE_TIMING
int read_phase_cycles(unsigned long long* out, int n, bool reset) {
  unsigned long long h[16];
  if (cudaMemcpyFromSymbol(h, g_phase_cycles, sizeof(h)) != cudaSuccess) return -1;
  for (int i = 0; i < n && i < 16; ++i) out[i] = h[i];
  if (reset) {
    unsigned long long z[16] = {0};
    if (cudaMemcpyToSymbol(g_phase_cycles, z, sizeof(z)) != cudaSuccess) return -1;
  }
  return 0;
}
#endif
void build_presieve_tables(uint32_t* out) {
  static const uint32_t groups[kPreGroups][3] = {{7, 11, 13}, {17, 19, 0}, {23, 29, 0}, {31, 0, 0}};
  for (int g = 0; g < kPreGroups; ++g) {
    const uint32_t P = kPreMod[g];
    for (uint32_t j = 0; j < P; ++j) {
      uint32_t m = 0xFFFFFFFFu;
      for (uint32_t jb = 0; jb < 4; ++jb)
        for (uint32_t o = 0; o < 8; ++o) {
          const uint64_t k = 4ull * j + jb;  // byte index modulo P
          for (int q = 0; q < 3 && groups[g][q]; ++q) {
            const uint32_t p = groups[g][q];
            if ((30ull * k + wheel_residue((int)o)) % p == 0) m &= ~(1u << (8 * jb + o));
          }
        }
      out[kPreOff[g] + j] = m;
    }
  }
}

size_t sieve_smem_bytes(uint32_t tile_words) {
  return (size_t)(tile_words + kSpareWords + kPreWords + kSmCounters) * sizeof(uint32_t);
}

// The largest dynamic shared memory of a kernel is an attribute of the device's function, which all
// contexts share: it goes to all that a block can have, whatever tile the calling context uses, so that no
// context lowers it for another.  A tile beyond it is refused without a failing CUDA call, whose error the next
// launch would report as its own.
template <int BLOCK, bool EMIT>
static int allow_smem(size_t smem) {
  auto fn = sieve_tiles_kernel<BLOCK, EMIT>;
  int dev = 0, most = 0;
  cudaFuncAttributes fa;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaFuncGetAttributes(&fa, fn) != cudaSuccess ||
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return -1;
  most -= (int)fa.sharedSizeBytes;
  if (smem > (size_t)std::max(most, 0)) return -1;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess ? 0 : -1;
}

template <int BLOCK>
static int block_attrs(size_t smem, int* max_ctas_per_sm) {
  if (allow_smem<BLOCK, false>(smem) || allow_smem<BLOCK, true>(smem)) return -1;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(max_ctas_per_sm, sieve_tiles_kernel<BLOCK, false>, BLOCK,
                                                       smem) == cudaSuccess
             ? 0
             : -1;
}

int sieve_kernel_attrs(int block, size_t smem, int* max_ctas_per_sm) {
  if (block == 512) return block_attrs<512>(smem, max_ctas_per_sm);
  if (block == 1024) return block_attrs<1024>(smem, max_ctas_per_sm);
  return -1;
}

int launch_sieve_stats(const SieveArgs& a, int grid, int block, size_t smem, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (block == 512) sieve_tiles_kernel<512, false><<<grid, 512, smem, s>>>(a);
  else if (block == 1024) sieve_tiles_kernel<1024, false><<<grid, 1024, smem, s>>>(a);
  else return -1;
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_sieve_emit(const SieveArgs& a, int grid, int block, size_t smem, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (block == 512) sieve_tiles_kernel<512, true><<<grid, 512, smem, s>>>(a);
  else if (block == 1024) sieve_tiles_kernel<1024, true><<<grid, 1024, smem, s>>>(a);
  else return -1;
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_tail(const SieveArgs& a, uint32_t max_tiles, IntervalOut* out, voss_interval_stats* stats,
                const uint32_t* out_index, void* stream, uint32_t* kernels) {
  if (a.n_intervals == 0) return 0;
  // one interval of few tiles: its block takes the seams along.  In a batch the intervals' numbers of
  // tiles differ by thousands, and a thread per tile evens them out.
  const bool stitched = a.n_tiles > 0 && (a.n_intervals > 1 || max_tiles > 8u * kTailBlock);
  if (stitched) stitch_kernel<<<(a.n_tiles + 255) / 256, 256, 0, (cudaStream_t)stream>>>(a);
  tail_kernel<<<a.n_intervals, kTailBlock, 0, (cudaStream_t)stream>>>(a, stitched, out, stats, out_index);
  *kernels += stitched ? 2 : 1;
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int probe_smem_rmw(int sm_count, void* stream, float* ms, double* bytes) {
  cudaStream_t s = (cudaStream_t)stream;
  const int grid = sm_count * 2;
  uint32_t* sink = nullptr;
  if (cudaMalloc(&sink, grid * sizeof(uint32_t)) != cudaSuccess) return -1;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  smem_rmw_probe_kernel<<<grid, 1024, 0, s>>>(sink);  // warm-up
  cudaEventRecord(e0, s);
  const int reps = 5;
  for (int r = 0; r < reps; ++r) smem_rmw_probe_kernel<<<grid, 1024, 0, s>>>(sink);
  cudaEventRecord(e1, s);
  cudaError_t st = cudaEventSynchronize(e1);
  float t = 0;
  cudaEventElapsedTime(&t, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(sink);
  if (st != cudaSuccess) return -1;
  *ms = t / reps;
  *bytes = (double)grid * 1024.0 * kProbeIters * 8.0;
  return 0;
}

}  // namespace voss
