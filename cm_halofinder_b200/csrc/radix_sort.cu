// Order of records by a 64-bit key: stable LSD radix sort of (key, index) pairs.
//
// The emission of the records has counted the digits of every pass, which
// gives each digit's start in the output (k_rs_offsets).  Each pass is then a single
// kernel: each 4096-key tile ranks its keys stably with warp ballot
// counters, learns how many keys of each digit the lower tiles hold by
// decoupled look-back over published tile states, stages its keys in shared
// memory in digit order and writes each digit's run contiguously
// (coalesced).  Only the order is wanted: the keys are
// narrowed to 32-bit words at the first pass after which at most 32 key
// bits remain (the consumed low digits are dropped), so that the later
// passes move 8 bytes per pair instead of 12; and those 32-bit passes use
// 9-bit digits where that saves a pass (26 bits: 9 + 9 + 8, not 8 + 8 + 8 + 2).
#include <algorithm>

#include "cmh_internal.cuh"

namespace cmh {
namespace {

constexpr int kTile = 4096;
constexpr int kBins = 256;      // 8-bit digits
constexpr int kMaxBins = kRadixBins;  // 9-bit digits
constexpr int kMaxPasses = kRadixPasses;
// Tile states of the look-back, one 64-bit word per (tile, digit): the flag
// in the high half, the count in the low half, written in one store.
constexpr uint64_t kAggregate = 1ull << 32;  // count = the tile's own keys of the digit
constexpr uint64_t kInclusive = 2ull << 32;  // count = keys of the digit up to this tile

template <int BINS = kBins, class K>
__device__ __forceinline__ uint32_t digit_of(K k, int shift) {
  return (uint32_t)(k >> shift) & (BINS - 1);
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}


// Where a pass reads its keys: an array, or a field of records `stride` bytes
// apart (their values are then the records' indices).
template <class K>
struct KeySource {
  const K *keys;
  uint32_t stride;  // bytes from one key to the next
  __device__ __forceinline__ K operator[](int64_t i) const {
    return *reinterpret_cast<const K *>(reinterpret_cast<const unsigned char *>(keys) +
                                        (uint64_t)i * stride);
  }
};

// Exclusive prefix over the digits of each pass (one CTA of kMaxBins
// threads per pass; unused digits count 0).
__global__ void __launch_bounds__(kMaxBins) k_rs_offsets(const uint32_t *__restrict__ ghist,
                                                         uint32_t *__restrict__ goff) {
  __shared__ uint32_t warp_sums[kMaxBins / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t v = ghist[blockIdx.x * kMaxBins + threadIdx.x];
  const uint32_t inc = warp_inclusive(v);
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < kMaxBins / 32 ? warp_sums[lane] : 0;
    const uint32_t wi = warp_inclusive(w);
    if (lane < kMaxBins / 32) warp_sums[lane] = wi - w;
  }
  __syncthreads();
  goff[blockIdx.x * kMaxBins + threadIdx.x] = inc - v + warp_sums[warp];
}

// One digit pass, single sweep: a CTA takes the next tile from a counter
// (so every lower tile is already being worked on), ranks its 4096 keys
// stably in shared memory (512 threads x 8 keys; warp match/ballot counters),
// publishes its per-digit counts, then finds the counts of all lower tiles
// by looking back through their published states (decoupled look-back:
// inclusive states end the walk) and writes each digit's run contiguously to
// goff[digit] + (keys of the digit in lower tiles).  A tile publishes its own
// counts before it waits on anything, so every wait ends; a wait is still
// capped, and a capped one sets *giveups.  The output then has holes of stale
// keys that the digit counts do not know, which a later pass would place past the
// arrays' ends: a CTA that finds *giveups set when it starts moves nothing.
constexpr int kSThreads = 512;
constexpr int kSWarps = kSThreads / 32;
constexpr int kSIPT = kTile / kSThreads;  // 8

// A tile in shared memory: its pairs in digit order, with the digits where the
// written keys no longer hold them, and 16-bit counters (a tile has 4096 keys;
// 32-bit ones cost the 9-bit passes a CTA per SM).
template <class KO, int BINS, bool NARROW>
struct ScatterSmem {
  KO keys[kTile];
  uint32_t vals[kTile];
  uint8_t digit[NARROW ? kTile : 4];
  uint16_t wcnt[kSWarps][BINS];
  uint32_t dstart[BINS];
  uint32_t gofs[BINS];
  uint32_t thist[BINS];
  uint32_t warp_sums[kSWarps];
  uint32_t tile, stop;
};

// Lanes of the warp with the same NB-bit value d (a digit, or BINS for an
// empty slot): one ballot per bit.
template <int NB>
__device__ __forceinline__ uint32_t peers_of(uint32_t d) {
  uint32_t peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < NB; b++) {
    const uint32_t m = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    peers &= ((d >> b) & 1u) ? m : ~m;
  }
  return peers;
}

__device__ __forceinline__ uint64_t load_state(const uint64_t *p) {
  return *reinterpret_cast<const volatile uint64_t *>(p);
}

// Keys are read as K and written as KO: K >> out_shift in a pass that narrows
// 64-bit keys to 32 bits (NARROW), K itself otherwise, and not at all in the last
// pass; digits have log2(BINS) bits.  Bound by instruction issue (ranking and
// staging).  256^3 box, 17.7M keys: 0.26 + 0.22 + 0.21 + 0.17 ms with 32-bit
// counters, whole keys staged in the narrowing pass and keys written in the last,
// 0.22 + 0.20 + 0.20 + 0.16 ms so; counts published after the ranking, which then
// needs no second histogram: 0.22 + 0.21 + 0.21 + 0.16.
template <class K, class KO, int BINS, bool NARROW, bool LAST>
__global__ void __launch_bounds__(kSThreads, NARROW || sizeof(KO) == 8 ? 3 : 4) k_rs_scatter(
    KeySource<K> keys_in, const uint32_t *__restrict__ vals_in,
    KO *__restrict__ keys_out, uint32_t *__restrict__ vals_out, int64_t n_cap,
    const uint32_t *__restrict__ n_dev, int shift, int out_shift,
    const uint32_t *__restrict__ goff,
    uint64_t *__restrict__ state, uint32_t *__restrict__ tile_ctr,
    unsigned int *__restrict__ giveups, SortWaits waits) {
  const int64_t n = n_dev ? (int64_t)*n_dev : n_cap;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Smem = ScatterSmem<KO, BINS, NARROW>;
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sm.tile = atomicAdd(tile_ctr, 1u);
  if (threadIdx.x == 32) sm.stop = __ldcg(giveups);  // (beside the other's wait)
  for (int i = threadIdx.x; i < kSWarps * BINS / 2; i += kSThreads)
    reinterpret_cast<uint32_t *>(&sm.wcnt[0][0])[i] = 0;
  if (threadIdx.x < BINS) sm.thist[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t tile = sm.tile;
  const int64_t base = (int64_t)tile * kTile;
  if (base >= n) return;  // the whole CTA leaves together
  if (sm.stop) {          // so too here, with an end to the higher tiles' waits
    if (threadIdx.x < BINS)
      atomicExch(reinterpret_cast<unsigned long long *>(state + (uint64_t)tile * BINS +
                                                        threadIdx.x),
                 (unsigned long long)kInclusive);
    return;
  }
  const uint32_t lt_mask = (1u << lane) - 1u;
  const int rem = n - base < kTile ? (int)(n - base) : kTile;
  const int mine = warp * 32 * kSIPT + lane;  // the thread's keys: mine + 32 j
  KO k[kSIPT];
  uint32_t v[kSIPT], dr[kSIPT];  // digit, later digit | rank << 16
#pragma unroll
  for (int j = 0; j < kSIPT; j++) {
    const int64_t i = base + mine + 32 * j;
    const bool valid = mine + 32 * j < rem;
    const K key = valid ? keys_in[i] : K(0);
    k[j] = NARROW ? (KO)(key >> out_shift) : (KO)key;
    dr[j] = valid ? digit_of<BINS>(key, shift) : (uint32_t)BINS;
    v[j] = valid ? (vals_in ? vals_in[i] : (uint32_t)i) : 0u;
  }
  // the tile's digit counts first, published before the ranking so that
  // the higher tiles' look-back finds them early
#pragma unroll
  for (int j = 0; j < kSIPT; j++)
    if (dr[j] < BINS) atomicAdd(&sm.thist[dr[j]], 1u);
  __syncthreads();
  // (a tile named by waits.stall_tile publishes nothing: a test hook whose
  // successor's capped wait then runs out)
  if (threadIdx.x < BINS && tile != waits.stall_tile)
    atomicExch(reinterpret_cast<unsigned long long *>(state + (uint64_t)tile * BINS + threadIdx.x),
               (unsigned long long)((tile == 0 ? kInclusive : kAggregate) | sm.thist[threadIdx.x]));
#pragma unroll
  for (int j = 0; j < kSIPT; j++) {
    const uint32_t d = dr[j];
    const bool valid = d < BINS;
    const uint32_t peers = peers_of<BINS == 512 ? 10 : 9>(d);
    const uint32_t lt = peers & lt_mask;
    uint32_t c = 0;
    if (valid) c = sm.wcnt[warp][d];
    __syncwarp();
    if (valid && lt == 0) sm.wcnt[warp][d] = (uint16_t)(c + __popc(peers));
    __syncwarp();
    dr[j] = d | (c + __popc(lt)) << 16;
  }
  __syncthreads();
  {
    // per digit: exclusive prefix over the warps, then over the digits
    const int d = threadIdx.x;
    uint32_t acc = 0;
    if (d < BINS) {
#pragma unroll
      for (int w = 0; w < kSWarps; w++) {
        const uint32_t t = sm.wcnt[w][d];
        sm.wcnt[w][d] = (uint16_t)acc;
        acc += t;
      }
    }
    uint32_t inc = warp_inclusive(acc);
    if (lane == 31) sm.warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = lane < kSWarps ? sm.warp_sums[lane] : 0;
      uint32_t wi = warp_inclusive(w);
      if (lane < kSWarps) sm.warp_sums[lane] = wi - w;
    }
    __syncthreads();
    if (d < BINS) {
      const uint32_t first = inc - acc + sm.warp_sums[warp];
      sm.dstart[d] = first;
      // add up the lower tiles' counts, then publish the running total
      uint64_t *own = state + (uint64_t)tile * BINS + d;
      uint32_t excl = 0;
      if (tile != 0) {
        for (int64_t j = (int64_t)tile - 1; j >= 0; j--) {
          const uint64_t *p = state + (uint64_t)j * BINS + d;
          uint64_t w = load_state(p);
          for (uint32_t spin = 0; (w >> 32) == 0 && spin < waits.spin_cap; spin++)
            w = load_state(p);
          if ((w >> 32) == 0) {
            atomicAdd(giveups, 1u);
            break;
          }
          excl += (uint32_t)w;
          if ((w >> 32) == 2) break;
        }
        if (tile != waits.stall_tile)
          atomicExch(reinterpret_cast<unsigned long long *>(own),
                     (unsigned long long)(kInclusive | (uint64_t)(excl + acc)));
      }
      sm.gofs[d] = goff[d] + excl - first;  // (modulo 2^32: first is added back below)
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSIPT; j++) {
    const uint32_t d = dr[j] & 0xffffu;
    if (d < BINS) {
      const uint32_t lp = sm.dstart[d] + sm.wcnt[warp][d] + (dr[j] >> 16);
      sm.keys[lp] = k[j];
      sm.vals[lp] = v[j];
      if constexpr (NARROW) sm.digit[lp] = (uint8_t)d;
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < rem; q += kSThreads) {
    const KO key = sm.keys[q];
    const uint32_t d = NARROW ? sm.digit[q] : digit_of<BINS>(key, shift);
    const uint32_t g = sm.gofs[d] + (uint32_t)q;
    if constexpr (!LAST) keys_out[g] = key;
    vals_out[g] = sm.vals[q];
  }
}

// A pass: its kernel and dynamic shared memory.
template <class K, class KO, int BINS, bool NARROW, bool LAST>
void scatter_pass(const void *keys, uint32_t stride, const uint32_t *vals, void *keys_out,
                  uint32_t *vals_out, int64_t n, const uint32_t *n_dev, int shift, int out_shift,
                  const uint32_t *goff, uint64_t *state, uint32_t *tile_ctr,
                  unsigned int *giveups, SortWaits waits, cudaStream_t s) {
  constexpr size_t smem = sizeof(ScatterSmem<KO, BINS, NARROW>);
  const int64_t ntiles = (n + kTile - 1) / kTile;
  k_rs_scatter<K, KO, BINS, NARROW, LAST><<<(unsigned)ntiles, kSThreads, smem, s>>>(
      KeySource<K>{static_cast<const K *>(keys), stride}, vals, static_cast<KO *>(keys_out),
      vals_out, n, n_dev, shift, out_shift, goff, state, tile_ctr, giveups, waits);
  CMH_LAUNCHED();
}

// Dynamic shared memory of every scatter instantiation, set once per device
// (never inside a graph capture).
template <class K, class KO, int BINS, bool NARROW> void set_smem() {
  const int bytes = (int)sizeof(ScatterSmem<KO, BINS, NARROW>);
  CMH_CUDA(cudaFuncSetAttribute(k_rs_scatter<K, KO, BINS, NARROW, false>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  CMH_CUDA(cudaFuncSetAttribute(k_rs_scatter<K, KO, BINS, NARROW, true>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

void set_scatter_smem(cudaStream_t s) {
  static bool done[64] = {};
  int dev = 0;
  CMH_CUDA(cudaGetDevice(&dev));
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CMH_CUDA(cudaStreamIsCapturing(s, &cs));
  if (dev >= 64 || done[dev] || cs != cudaStreamCaptureStatusNone) return;
  set_smem<uint64_t, uint64_t, kBins, false>();
  set_smem<uint64_t, uint32_t, kBins, true>();
  set_smem<uint32_t, uint32_t, kBins, false>();
  set_smem<uint32_t, uint32_t, kMaxBins, false>();
  done[dev] = true;
}

// The passes of a sort of `bits`-bit keys: m 8-bit passes over the 64-bit keys,
// m the fewest (at least one) after which at most 32 bits remain, then the
// 32-bit passes over the R bits left, with 9-bit digits on the first
// R - 8 ceil(R / 9) of them when that takes fewer passes than 8-bit digits.
// *wide receives m.
PassDigits plan_passes(int bits, int *wide) {
  PassDigits pd{};
  const int m = std::max(1, std::min((bits + 7) / 8, (bits - 32 + 7) / 8));
  const int rest = std::max(0, bits - 8 * m);
  const int q8 = (rest + 7) / 8, q9 = (rest + 8) / 9;
  const int q = std::min(q8, q9), nine = q9 < q8 ? rest - 8 * q9 : 0;
  pd.passes = m + q;
  int shift = 0;
  for (int p = 0; p < pd.passes; p++) {
    pd.shift[p] = shift;
    pd.width[p] = (p >= m && p - m < nine) ? 9 : 8;
    shift += pd.width[p];
  }
  *wide = m;
  return pd;
}

}  // namespace

bool radix_states_apart(int64_t n, int bits, size_t *bytes) {
  int m = 0;
  const PassDigits pd = plan_passes(bits, &m);
  const int64_t ntiles = (std::max<int64_t>(n, 1) + kTile - 1) / kTile;
  size_t all = 0;
  for (int p = 0; p < pd.passes; p++) all += ((size_t)ntiles << pd.width[p]) * sizeof(uint64_t);
  const bool apart = all <= (64u << 20);
  *bytes = apart ? all : (size_t)ntiles * kMaxBins * sizeof(uint64_t);
  return apart;
}

PassDigits radix_order_plan(int bits) {
  int m = 0;
  return plan_passes(bits, &m);
}

void radix_order_records(const void *records, uint32_t stride, uint32_t key_at, uint64_t *keys_a,
                         uint32_t *vals_a, uint64_t *keys_b, uint32_t *vals_b, int64_t n,
                         const uint32_t *n_dev, int bits, RadixTmp tmp, unsigned int *giveups,
                         cudaStream_t s, SortWaits waits) {
  int m = 0;
  const PassDigits pd = plan_passes(bits, &m);
  if (bits > 64 || pd.passes > kMaxPasses)
    fail(CMH_ERR_INVALID_ARGUMENT, "radix sort: key bits out of range");
  const int64_t ntiles = (n + kTile - 1) / kTile;
  if (ntiles >= 0xffffffffll) fail(CMH_ERR_CAPACITY, "radix sort: too many tiles");
  uint64_t *state = tmp.state;
  uint32_t *ghist = tmp.counts;  // digit counts | digit offsets | tile counters
  uint32_t *goff = ghist + kMaxPasses * kMaxBins;
  uint32_t *tile_ctr = goff + kMaxPasses * kMaxBins;
  set_scatter_smem(s);
  k_rs_offsets<<<pd.passes, kMaxBins, 0, s>>>(ghist, goff);
  CMH_LAUNCHED();
  // the first pass reads the records (their indices are the values) and writes
  // the b buffers, the next the a buffers, and so on in turn; pass m - 1 writes
  // key >> 8 m as 32-bit words and the later passes sort those
  const void *src_k = static_cast<const unsigned char *>(records) + key_at;
  const uint32_t *src_v = nullptr;
  uint32_t src_stride = stride;
  void *out_k[2] = {keys_b, keys_a};
  uint32_t *out_v[2] = {vals_b, vals_a};
  for (int p = 0; p < pd.passes; p++) {
    const int bins = 1 << pd.width[p];
    if (!tmp.apart)
      CMH_CUDA(cudaMemsetAsync(state, 0, (size_t)ntiles * bins * sizeof(uint64_t), s));
    const uint32_t *go = goff + p * kMaxBins;
    void *dst_k = out_k[p % 2];
    uint32_t *dst_v = out_v[p % 2];
    // the stall hook applies to the first pass only
    const SortWaits wp{waits.spin_cap, p == 0 ? waits.stall_tile : 0xffffffffu};
    const bool last = p == pd.passes - 1;
    auto run = [&](auto pass, auto last_pass) {
      (last ? last_pass : pass)(src_k, src_stride, src_v, dst_k, dst_v, n, n_dev,
                                p < m ? pd.shift[p] : pd.shift[p] - 8 * m, 8 * m, go, state,
                                tile_ctr + p, giveups, wp, s);
    };
    if (p < m - 1)
      run(scatter_pass<uint64_t, uint64_t, kBins, false, false>,
          scatter_pass<uint64_t, uint64_t, kBins, false, true>);
    else if (p < m)
      run(scatter_pass<uint64_t, uint32_t, kBins, true, false>,
          scatter_pass<uint64_t, uint32_t, kBins, true, true>);
    else if (bins == kMaxBins)
      run(scatter_pass<uint32_t, uint32_t, kMaxBins, false, false>,
          scatter_pass<uint32_t, uint32_t, kMaxBins, false, true>);
    else
      run(scatter_pass<uint32_t, uint32_t, kBins, false, false>,
          scatter_pass<uint32_t, uint32_t, kBins, false, true>);
    src_stride = p < m - 1 ? sizeof(uint64_t) : sizeof(uint32_t);
    if (tmp.apart) state += (size_t)ntiles * bins;
    src_k = dst_k;
    src_v = dst_v;
  }
}

}  // namespace cmh
