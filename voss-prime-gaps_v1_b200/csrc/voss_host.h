// voss_host.h — host-runtime types shared by the C ABI (voss_api.cpp) and the request server
// (voss_server.cpp).  Not installed; the public interface is include/voss.h.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <mutex>
#include <thread>
#include <vector>

#include "voss.h"
#include "voss_internal.h"

namespace voss_host {

// Record a message for voss_last_error() and return `code`.
int fail(int code, const char* fmt, ...);

// NVTX range in the "voss" domain for the lifetime of the object: every API call and its host
// stages (plan, launch, sort, copy) show as named spans on an Nsight Systems timeline.  NVTX 3
// is header-only; with no tool attached a push/pop is a test of one pointer.
inline nvtxDomainHandle_t nvtx_domain() {
  static nvtxDomainHandle_t d = nvtxDomainCreateA("voss");
  return d;
}
struct NvtxRange {
  explicit NvtxRange(const char* name) {
    nvtxEventAttributes_t a = {};
    a.version = NVTX_VERSION;
    a.size = NVTX_EVENT_ATTRIB_STRUCT_SIZE;
    a.messageType = NVTX_MESSAGE_TYPE_ASCII;
    a.message.ascii = name;
    nvtxDomainRangePushEx(nvtx_domain(), &a);
  }
  ~NvtxRange() { nvtxDomainRangePop(nvtx_domain()); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

#define CUDA_TRY(call)                                                                      \
  do {                                                                                      \
    cudaError_t e__ = (call);                                                               \
    if (e__ != cudaSuccess)                                                                 \
      return ::voss_host::fail(VOSS_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e__)); \
  } while (0)

// A grow-only device buffer.
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
  int ensure(size_t need);
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// Device memory of one launch of the tile kernel (and of Miller-Rabin batches).
struct Workspace {
  DevBuf state;  // counters, IntervalOut and accumulators of a launch (state_of), zeroed and read as one
  DevBuf desc;   // what a launch copies in: intervals, pre-pass intervals, interval of each tile
  DevBuf partials, large, large_iv, over, istats, offsets, emit, mr_in, mr_out;
  DevBuf gbm;    // large-prime bitmap of the launch
  DevBuf pg_pa, pg_gap, pg_ok;  // gap proofs: inputs and verdicts (endpoints use mr_in / mr_out)
  DevBuf sha_data, sha_off, sha_out;  // certificate hashing: messages, offsets, digests
  DevBuf ls_keys, ls_idx, ls_temp, ls_sorted;  // large-gap list sorted by position (large_sort.cu)
  DevBuf sh_iv, sh_map, sh_seg;  // short intervals by Miller-Rabin (short_iv.cu); sieved intervals' result slots
  // Largest large-prime bitmap this workspace may use; with gbm_fixed the buffers are never
  // grown (server slots size them at creation), and launches that need more skip the pre-pass.
  size_t gbm_budget = 8ull << 30;
  bool gbm_fixed = false;
};

// Events bracketing one launch: ev0 before all of its device work (descriptor copies, memsets),
// ev1 after the tile kernel, ev2 after the kernels that close the launch (seams, results, the sort of a
// short gap list, the short-interval route); evp (optional) after the large-prime pre-pass, just before
// the tile kernel.
struct LaunchEvents {
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr, evp = nullptr;
};

// How a launch cuts its intervals into tiles and its base primes into categories.
struct TileShape {
  uint32_t chunk_words = 0;  // 32-bit words per thread of a tile
  uint32_t coop_div = 0;     // as voss_tuning
  uint32_t p_large = 0;      // primes from here on belong to the pre-pass
};

struct RunPlan {
  std::vector<voss::IntervalDev> iv;
  TileShape shape;
  uint32_t n_tiles = 0;
  uint64_t n_words = 0;
};

enum { kCtrTile = 0, kCtrLarge = 1, kCtrOver = 2, kCtrError = 3, kCtrWords = 8 };

constexpr size_t kCtrBytes = 64;  // counters at the front of Workspace::state
// The parts of Workspace::state in a launch of n intervals.
struct LaunchState {
  uint32_t* ctr;
  voss::IntervalOut* out;
  unsigned long long* acc;
  size_t bytes;
};
inline LaunchState state_of(const Workspace& W, size_t n) {
  char* p = static_cast<char*>(W.state.p);
  const size_t acc = kCtrBytes + sizeof(voss::IntervalOut) * n;
  return LaunchState{reinterpret_cast<uint32_t*>(p), reinterpret_cast<voss::IntervalOut*>(p + kCtrBytes),
                     reinterpret_cast<unsigned long long*>(p + acc),
                     acc + sizeof(unsigned long long) * voss::kAccStride * n};
}
inline size_t state_bytes(size_t n) {
  return kCtrBytes + (sizeof(voss::IntervalOut) + sizeof(unsigned long long) * voss::kAccStride) * n;
}
// Bytes of Workspace::desc: n intervals, n_scat pre-pass intervals, n_tiles tiles.
inline size_t desc_bytes(size_t n, size_t n_scat, size_t n_tiles) {
  return ((sizeof(voss::IntervalDev) * n + 15) & ~(size_t)15) + sizeof(voss::IntervalScatter) * n_scat +
         sizeof(uint32_t) * n_tiles;
}
// Records of the sorted large-gap list that come to the host together with the state.
constexpr uint32_t kFetchRecords = 4096;
constexpr size_t kFetchBytes = 128u << 10;  // voss_ctx::h_fetch

constexpr uint64_t kMaxHi = 1ull << 62;
constexpr uint32_t kOverCap = 1u << 16;
constexpr uint64_t kDefaultLargeCap = 1ull << 22;
// Large-prime pre-pass windows: bitmap bytes per window, inside the 126 MB L2 next to the primes
// the pre-pass reads (23 MB of 32-bit primes below 10^8).  The 4096-interval batch's pre-pass takes 7.8 ms
// with 48 MB, 8.5, 8.1, 8.0 and 8.1 ms with 16, 24, 32 and 64 MB; the 157 MB bitmap of 4.7e9 integers
// near 10^15 1.30 ms in four pieces against 4.24 ms in one.
#ifndef VOSS_SCATTER_WINDOW_MB
#define VOSS_SCATTER_WINDOW_MB 48
#endif
constexpr uint64_t kScatterWindowBytes = (uint64_t)VOSS_SCATTER_WINDOW_MB << 20;
constexpr uint64_t kScatterWindowWords = kScatterWindowBytes / 4;
// Large host transfers: bytes per chunk through a pinned buffer, bytes per copying host thread at
// least, and Miller-Rabin candidates per chunk.  10^7 candidates take 3.5 ms per call at 2^20 per
// chunk, 4.2 at 2^19 and 4.2 at 2^21 (6.3 ms in one chunk); 6*10^6 primes (48 MB) 3.7 ms in 8 MB
// chunks, 4.9 in 4 MB, 3.7 in 16 MB (11.5 ms straight to pageable memory).
constexpr size_t kStageChunk = 8u << 20;
constexpr size_t kStagePart = 1u << 20;
constexpr uint64_t kMrChunk = 1ull << 20;
constexpr uint64_t kMaxLargeCap = 50000000ull;  // MAX_LARGE_GAPS, src/voss_v7_live.cu:34

}  // namespace voss_host

struct voss_ctx {
  int device = 0;
  int sm_count = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t copy_stream = nullptr;  // host-to-device copies overlapped with work on `stream`
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr, evp = nullptr;
  uint64_t max_hi = 0;
  std::vector<uint32_t> primes;  // >= 37
  voss_host::DevBuf d_primes, d_magic, d_pretab;
  voss_host::DevBuf d_cls_primes, d_cls_inv, d_cls_index;  // the primes below kClsLimit by class (SieveArgs)
  uint32_t cls_first[8] = {0};
  uint32_t n_cls_blocks = 0;
  voss_tuning tune{};
  bool auto_shape = true;  // the tile shape was left to the library: small launches choose their own
  int ctas_per_sm = 1;
  voss_host::Workspace ws;
  // last range run
  bool have_range = false;
  uint64_t r_lo = 0, r_hi = 0, r_seg = 0;
  uint32_t r_flags = 0;
  uint32_t r_tiles = 0;
  uint64_t r_large_cap = 0;
  float sieve_ms = 0, total_ms = 0;
  uint32_t last_kernels = 0;  // kernels of the last launch (with the short-interval route's)
  // host side of the large-gap list: pinned, grow-only staging for the device-to-host copy of
  // the list (sorted on the device), so that repeated calls touch no fresh pages
  voss_large_gap* h_large = nullptr;
  // pinned: the state of a one-interval launch and the first kFetchRecords large gaps, or a small result
  char* h_fetch = nullptr;
  size_t h_large_cap = 0;
  // pinned staging of large host batches (Miller-Rabin candidates in, verdicts out): two
  // buffers, one filled by host threads while the other crosses; ev_stage[b] marks the end of
  // buffer b's last transfer
  uint64_t* h_stage[2] = {nullptr, nullptr};
  size_t h_stage_cap = 0;  // 64-bit entries per buffer
  cudaEvent_t ev_stage[2] = {nullptr, nullptr};
  cudaEvent_t ev_out[2] = {nullptr, nullptr};  // a Miller-Rabin chunk's verdicts are in buffer b
  // most 64-bit entries a staging buffer may hold (larger transfers cross in chunks); the
  // environment variable VOSS_STAGE_LIMIT lowers it when the context is created, so tests can
  // drive the chunked paths with small batches
  size_t stage_limit = ~(size_t)0;
};

namespace voss_host {

// The context's tile shape.
TileShape default_shape(const voss_ctx* c);
// The shape for a launch of these intervals (at most max_tiles tiles, 0: no limit): the context's,
// or a smaller one when the launch would leave SMs idle.
TileShape choose_shape(const voss_ctx* c, const uint64_t* lo, const uint64_t* hi, uint32_t n, uint64_t max_tiles);
// Cut intervals [lo_i, hi_i) into tiles; intervals without wheel integers get no tiles.
int plan_intervals(const voss_ctx* c, const uint64_t* lo, const uint64_t* hi, uint32_t n, uint64_t seg_k,
                   const TileShape& shape, RunPlan* P);
// Queue plan P on stream s, using the workspace W and events E: the tile kernel, and unless emit the
// tail (with `stats`: of interval statistics at stats[out_index[i]]).  *kernels: how many ran.
int launch_plan_ws(voss_ctx* c, Workspace& W, const LaunchEvents& E, const RunPlan& P, bool want_large,
                   uint64_t large_cap, bool emit, cudaStream_t s, uint32_t min_gap, voss_interval_stats* stats,
                   const uint32_t* out_index, uint32_t* kernels);
// A batch of intervals split between the sieve (lo, hi, map = their positions in the batch)
// and the Miller-Rabin path for short intervals at high starts (sv, n_cand candidates).
struct IntervalRoute {
  std::vector<uint64_t> lo, hi;
  std::vector<uint32_t> map;
  std::vector<voss::ShortInterval> sv;
  uint64_t n_cand = 0;
  uint32_t n_seg = 0;  // segments of the Miller-Rabin intervals
};
// Split [lo_i, hi_i) by the context's mr_route, with at most cand_cap Miller-Rabin candidates.
void route_intervals(const voss_ctx* c, const uint64_t* lo, const uint64_t* hi, uint32_t n, uint64_t cand_cap,
                     IntervalRoute* R);
// Launch a routed batch of n intervals on stream s; all n results land in W.istats (lo, hi and
// the primes 2, 3, 5 are the host's, add_small_primes).  E.ev2 is recorded after the last kernel.
int launch_routed(voss_ctx* c, Workspace& W, const LaunchEvents& E, const IntervalRoute& R, uint32_t n,
                  cudaStream_t s, uint32_t* kernels);
int check_device_error(const uint32_t* ctr_host);
// memcpy split over up to 8 host threads, in parts of at least min_part bytes.
void parallel_copy(void* dst, const void* src, size_t bytes, size_t min_part = 8u << 20);
// Up to 8 host threads that copy together for the duration of one call: a chunked transfer starts
// them once (a thread costs tens of microseconds) and hands them each chunk.
class CopyTeam {
 public:
  explicit CopyTeam(size_t total_bytes);  // a thread per kStagePart bytes at most
  ~CopyTeam();
  CopyTeam(const CopyTeam&) = delete;
  CopyTeam& operator=(const CopyTeam&) = delete;
  void copy(void* dst, const void* src, size_t bytes);  // memcpy, returns when all of it is done

 private:
  void work(size_t i);
  void copy_part(size_t i) const;
  void post();
  std::vector<std::thread> th_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::atomic<uint64_t> job_{0};
  std::atomic<size_t> left_{0};
  bool stop_ = false;  // written before the last post()
  void* dst_ = nullptr;
  const void* src_ = nullptr;
  size_t bytes_ = 0;
};
struct CopySeg {
  const void* src;
  size_t bytes;
};
// The segments copied back to back into dst, split the same way.
void parallel_gather(void* dst, const CopySeg* seg, size_t n_seg, size_t min_part);
std::vector<uint64_t> small_primes_in(uint64_t lo, uint64_t hi);
// Add the primes 2, 3, 5 of [lo, hi) to a device-finalized interval result.
void add_small_primes(voss_interval_stats& st, uint64_t lo, uint64_t hi);

}  // namespace voss_host
