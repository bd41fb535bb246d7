// Internal declarations of the B200 FoF library (not part of the C ABI).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/cmh_fof.h"

namespace cmh {

constexpr int kSMs = 148;  // B200: 2 dies x 74 SMs

// Per-thread error message behind cmh_last_error().
void set_error(const std::string &msg);

struct Error {
  cmh_status code;
  std::string msg;
};

// Throws Error on a CUDA failure; the C ABI layer turns it into a status.
void cuda_check(cudaError_t e, const char *what, const char *file, int line);
#define CMH_CUDA(x) ::cmh::cuda_check((x), #x, __FILE__, __LINE__)

// Kernels launched by this host thread (reported per run in cmh_stats).
extern thread_local long long g_launches;
#define CMH_LAUNCHED()                     \
  do {                                     \
    CMH_CUDA(cudaGetLastError());          \
    ++::cmh::g_launches;                   \
  } while (0)
[[noreturn]] void fail(cmh_status code, const std::string &msg);

// Host-side fault injection for tests: whether `kind` is one of the
// comma-separated words of the CMH_FAULT environment variable (alloc: device
// allocations fail; io: opening a file fails; overflow: every run overflows
// its capacity; lookback: one tile of the cell sort publishes nothing, so a
// capped device wait runs out; gather: the same of the run count).  Read on every call, in host code only.
bool fault_active(const char *kind);

// Grid size for a grid-stride kernel: a multiple of the SM count, capped by
// the work.
inline unsigned grid_for(int64_t n, int threads, int per_sm = 8) {
  int64_t want = (n + threads - 1) / threads;
  int64_t cap = (int64_t)kSMs * per_sm;
  if (want < 1) want = 1;
  return (unsigned)(want < cap ? want : cap);
}

// CTAs of `kernel` (with `threads` threads and `smem` bytes of dynamic shared
// memory) resident at once on the current device: per-SM occupancy times the
// SM count, cached per kernel, shape and device.
int resident_ctas(const void *kernel, int threads, size_t smem);

// Grid for a grid-stride kernel: one resident wave, capped by the work.
inline unsigned grid_resident(const void *kernel, int threads, size_t smem, int64_t n) {
  int64_t want = (n + threads - 1) / threads;
  const int64_t cap = resident_ctas(kernel, threads, smem);
  if (want < 1) want = 1;
  return (unsigned)(want < cap ? want : cap);
}

// Growable device buffer, or a piece of another one (a view).
struct DevBuf {
  void *p = nullptr;
  size_t cap = 0;
  bool view = false;
  void ensure(size_t bytes);
  void place(const DevBuf &in, size_t at, size_t bytes);
  void release();
  template <class T> T *as() const { return reinterpret_cast<T *>(p); }
};

// ---- radix_sort.cu -----------------------------------------------------------
// Bounds of the look-back waits (the sort's and the run count's): a tile polls
// a lower tile's state at most spin_cap times, then gives up (the run's giveups
// counter is raised; a sort's output is then not an ordering).  stall_tile (a
// test hook) names a tile (of a sort's first pass) that publishes nothing, so
// that its successor's wait runs out.
constexpr uint32_t kSpinCap = 1u << 22;
struct SortWaits {
  uint32_t spin_cap = kSpinCap;
  uint32_t stall_tile = 0xffffffffu;
};

// The digits of a sort's passes: shift in the original key and width (8 or
// 9 bits); pass p's digit counts take kRadixBins words from kRadixBins p on.
constexpr int kRadixBins = 512;
constexpr int kRadixPasses = 8;
struct PassDigits {
  int passes;
  int shift[kRadixPasses];
  int width[kRadixPasses];
};

// The order of n records by the low `bits` bits (at least one pass is made) of
// a 64-bit key that each holds `key_at` bytes in: the records' indices, in
// stable key order, end in vals_b after an odd number of passes, else in
// vals_a.  Both key buffers are scratch: the first pass reads the records and
// their indices need no array, and the later passes move 32-bit key words,
// with 9-bit digits where that saves a pass.
// The caller counts the digits of radix_order_plan(bits) of all records into
// the counts as it writes them.
// `n` sizes the launches; with `n_dev` set, the element count is read from
// device memory (at most n), so the sort needs no host synchronisation.
// `giveups` (device) counts capped look-back waits.
//
// Scratch: kRadixCounts cleared words of digit counts (and what follows from
// them), and the tiles' look-back states: the bytes that radix_states_apart
// gives.  Where it returns true (up to 64 MB in all) every pass has its own and
// the caller clears them; else the sort clears them before each pass.
constexpr int kRadixCounts = 2 * kRadixPasses * kRadixBins + kRadixPasses;
struct RadixTmp {
  uint64_t *state;
  uint32_t *counts;
  bool apart;
};
bool radix_states_apart(int64_t n, int bits, size_t *bytes);
PassDigits radix_order_plan(int bits);
void radix_order_records(const void *records, uint32_t stride, uint32_t key_at, uint64_t *keys_a,
                         uint32_t *vals_a, uint64_t *keys_b, uint32_t *vals_b, int64_t n,
                         const uint32_t *n_dev, int bits, RadixTmp tmp, unsigned int *giveups,
                         cudaStream_t s, SortWaits waits = SortWaits{});
}  // namespace cmh
