// The FoF hot path on one B200: ingest + periodic images, cell keys, radix
// sort, fine-cell runs, befriending with a lock-free union-find, and the
// segmented reductions that produce the halo catalog.  A run holds one or
// many independent domains ("boxes"); all of them go through the same
// launches (one sort, one befriending pass, one reduction for the batch), and
// no size is read back by the host until the run is issued, so a run can be
// captured in a CUDA graph and replayed.
//
// Reference: src_v2/FOF.c (FOF, Befriend, Checkhalo, Output_Halos property
// sums) and src_v2/read_data.c:409-424,785-816 (domain filter, ghost wrap).
//
// Cells.  Particles are keyed by a fine cell of side h <= l_min / sqrt(3)
// (with a 2^-20 margin): two particles in the same fine cell are closer than
// the linking length whatever their position inside it, so every occupied
// fine cell is one connected piece and union-find runs over cells, not
// particles.  Fine cells are grouped k^3 to a top cell; the sort key is
// (top cell, fine cell inside it), each box's top cells numbered after the
// previous box's, so a top cell's fine cells are contiguous and the
// befriending step visits the 27-cell top stencil (self + 13 forward
// neighbours), exactly the cell loop of FOF.c:96-161 one level up.
//
// Pair predicate.  A pair of particles is linked iff the reference's double
// expression ((dx*dx + dy*dy) + dz*dz) <= Linklength^2 holds (FOF.c:351-357),
// dx being a float subtraction for float positions (MEMORY_MODE).
// CMH_PLAIN_FP64 evaluates exactly that for every pair.  CMH_FP32_RECHECK
// evaluates d2_32 = fma(dz,dz, fma(dy,dy, dx*dx)) in FP32 and re-tests in
// double only when t_lo <= d2_32 <= t_hi.  Band proof, float positions:
//   dx is the same float in both paths.  With u = 2^-24 and D the exact sum
//   of the three (exactly representable in double) squares,
//   |d2_32 - D| <= g3 D (g3 = 3u/(1-3u): each term sees at most three
//   roundings), and the reference's value d2_64 = D (1 + t), |t| <= 2^-52.
//   t_lo = fl32(l2) - 4 ulp, with |fl32(l2) - l2| <= ulp/2 and ulp > u l2,
//   so d2_32 < t_lo gives D < l2 (1 - 3.5u) / (1 - g3) < l2 (1 - 0.4u) and
//   hence d2_64 < l2: linked.  Symmetrically d2_32 > t_hi gives d2_64 > l2.
//   For double positions dx_32 = fl32(dx_64) adds 2u, and the band is 8 ulp.
//   Subnormal squares add at most 3 * 2^-149 in absolute terms, far below
//   the 0.4u l2 margin for any linking length above 1e-15.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "cmh_internal.cuh"
#include "fof_kernels.cuh"
#include "plan.cuh"

namespace cmh {

namespace {

constexpr int kT = 256;              // threads per block for element-wise kernels
constexpr uint32_t kNone = 0xffffffffu;
constexpr uint64_t kM21 = (1ull << 21) - 1;

__constant__ int kFwd[14][3] = {
    {0, 0, 0},                                                   // self
    {1, 0, 0},   {-1, 1, 0}, {0, 1, 0},  {1, 1, 0},              // same z
    {-1, -1, 1}, {0, -1, 1}, {1, -1, 1}, {-1, 0, 1}, {0, 0, 1},  // z + 1
    {1, 0, 1},   {-1, 1, 1}, {0, 1, 1},  {1, 1, 1}};

__device__ __forceinline__ int64_t gtid() {
  return (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
}
__device__ __forceinline__ int64_t gstride() { return (int64_t)gridDim.x * blockDim.x; }

template <class T> __device__ __forceinline__ double as_d(T v) { return (double)v; }

// Index of the last entry of base[0..nb) that is <= x (base[0] == 0).
__device__ __forceinline__ int box_search(const uint64_t *base, int nb, uint64_t x) {
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= x) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Copies the boxes' first input index (or first top cell) into shared memory.
__device__ __forceinline__ void load_bases(const BoxDev *boxes, int nbox, uint64_t *s, bool tops) {
  for (int b = threadIdx.x; b < nbox; b += blockDim.x) s[b] = tops ? boxes[b].top_base : boxes[b].in_base;
  __syncthreads();
}

// Fills of the later stages' tables, one launch for all: 16 bytes per store,
// every array's room being a multiple of that (a node per array delayed the
// ingest's first kernel in a replayed graph: 64^3 box 0.37 ms a pass, 0.31 with one).
struct Fills {
  static constexpr int kMax = 16;
  uint4 *p[kMax];
  uint64_t n[kMax];     // 16-byte words
  uint32_t word[kMax];  // what every 4 bytes are set to
  int count = 0;
  void add(const DevBuf &b, size_t bytes, uint32_t w) {
    if (bytes == 0) return;
    if (count == kMax) fail(CMH_ERR_CAPACITY, "too many tables to fill");  // (14 at most)
    p[count] = b.as<uint4>();
    n[count] = (bytes + 15) / 16;
    word[count++] = w;
  }
};

__global__ void __launch_bounds__(kT) k_fill(const __grid_constant__ Fills f) {
  for (int q = 0; q < f.count; q++) {
    const uint32_t w = f.word[q];
    const uint4 v = make_uint4(w, w, w, w);
    uint4 *p = f.p[q];
    for (uint64_t i = (uint64_t)gtid(); i < f.n[q]; i += (uint64_t)gstride()) p[i] = v;
  }
}

// ---------------------------------------------------------------------------
// Ingest: domain filter (read_data.c:409-424) and periodic images.
// ---------------------------------------------------------------------------

// Image shift s in {-1, +1} along axis a: the stored coordinate (the
// reference's wrap, read_data.c:792-797).
template <class PT>
__device__ __forceinline__ PT image_coord(const Geom &g, PT x, int a, int s) {
  return (PT)__dadd_rn((double)x, s > 0 ? g.L[a] : -g.L[a]);
}

template <class PT>
__device__ __forceinline__ void load_pos(const BoxDev &bx, uint64_t li, double x[3]) {
  const PT *pos = static_cast<const PT *>(bx.pos);
  x[0] = as_d(pos[3 * li]);
  x[1] = as_d(pos[3 * li + 1]);
  x[2] = as_d(pos[3 * li + 2]);
}

// Whether a particle at x is inside the domain (bit 6; NaN is outside) and
// which of its shifts stay in the shell (bit 2 a: by -L along axis a, bit
// 2 a + 1: by +L).  Comparisons in the position type only: the thresholds are
// exact, and the double arithmetic of every particle's shifts bounded the
// former count kernel.
template <class PT> struct IngestBox {
  PT dom_lo[3], dom_hi[3], img_lo[3], img_hi[3];
  float zmin, scale;
  uint32_t base, top;
  __device__ __forceinline__ explicit IngestBox(const BoxDev &bx) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      dom_lo[a] = (PT)bx.g.dom_lo[a];
      dom_hi[a] = (PT)bx.g.dom_hi[a];
      img_lo[a] = (PT)bx.g.img_lo[a];
      img_hi[a] = (PT)bx.g.img_hi[a];
    }
    zmin = (float)bx.g.rmin[2];
    scale = bx.bucket_scale;
    base = bx.bucket_base;
    top = bx.nbucket - 1u;
  }
  __device__ __forceinline__ uint32_t opts(const PT (&x)[3]) const {
    bool in = true;
    uint32_t o = 64u;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      in &= x[a] >= dom_lo[a] && x[a] <= dom_hi[a];
      o |= (x[a] >= img_lo[a] ? 1u : 0u) << (2 * a) | (x[a] <= img_hi[a] ? 2u : 0u) << (2 * a);
    }
    return in ? o : 0u;
  }
  // (the count and the emission agree on it; it need not follow the key exactly)
  __device__ __forceinline__ uint32_t bucket(PT z) const {
    const int q = __float2int_rd(__fmul_rn(__fsub_rn((float)z, zmin), scale));
    return base + min((uint32_t)max(q, 0), top);
  }
};

// Positions along axis a that a particle takes (itself and its images).
__device__ __forceinline__ uint32_t opt_count(uint32_t opts, int a) {
  return 1u + ((opts >> (2 * a)) & 1u) + ((opts >> (2 * a + 1)) & 1u);
}
// Records of an inside particle: itself and its images.
__device__ __forceinline__ uint32_t opt_records(uint32_t opts) {
  return opt_count(opts, 0) * opt_count(opts, 1) * opt_count(opts, 2);
}

// Ingest tiles: 256 PER consecutive particles of one box, PER per thread: four,
// or one while that leaves SMs without a tile (a lone tile is a chain of waits;
// 10,007 particles: 21 us of kernels in tiles of 1024, 17 us in tiles of 256).
// Buckets: slabs of a box, in the keys' order (z first).  The
// records are emitted bucket by bucket, so that the cell-ordered gather, whose
// consecutive elements come from one bucket, reads memory that is in L2
// (each 64 bytes it fetches are used up), not the whole array at random.  The
// order inside a bucket does not matter: the sort follows, and the processing
// indices are computed, not implied by the place.  Gather of the 256^3 box: 0.43
// ms at random, 0.24 ms by buckets; ingest 0.60 ms with whole-array flags and
// scans, 0.42 ms with tile sums.
constexpr int kPer = 4;
constexpr int kMaxBuckets = kMaxBoxes + 512;

// Box of an ingest tile (the last with tile_base <= tile and particles).
__device__ __forceinline__ int tile_box(const BoxDev *boxes, int nbox, uint32_t tile) {
  int lo = 0, hi = nbox - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (boxes[mid].tile_base <= tile) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A thread's PER consecutive particles from i on: 16-byte loads where the
// array is aligned and they come out even.
template <class PT, int PER>
__device__ __forceinline__ void load_some(const BoxDev &bx, uint64_t i, PT (&x)[PER][3]) {
  const PT *pos = static_cast<const PT *>(bx.pos) + 3 * i;
  constexpr int kBytes = 3 * PER * (int)sizeof(PT);
  if (kBytes % 16 == 0 && i + PER <= bx.n && ((uintptr_t)pos & 15) == 0) {
    __align__(16) PT v[3 * PER];
#pragma unroll
    for (int q = 0; q < kBytes / 16; q++)
      reinterpret_cast<uint4 *>(v)[q] = __ldg(reinterpret_cast<const uint4 *>(pos) + q);
#pragma unroll
    for (int j = 0; j < PER; j++)
#pragma unroll
      for (int a = 0; a < 3; a++) x[j][a] = v[3 * j + a];
  } else {
#pragma unroll
    for (int j = 0; j < PER; j++)
#pragma unroll
      for (int a = 0; a < 3; a++) x[j][a] = i + j < bx.n ? pos[3 * j + a] : PT(0);
  }
}

// Per tile the kept particles and their images, and the records per bucket.
template <class PT, int PER>
__global__ void __launch_bounds__(kT) k_ingest_count(const BoxDev *__restrict__ boxes, int nbox,
                                                     uint32_t ntile, int nbucket,
                                                     uint2 *__restrict__ tile_sum,
                                                     uint32_t *__restrict__ bucket_count) {
  __shared__ uint32_t s_bucket[kMaxBuckets];
  __shared__ uint32_t s_warp[kT / 32];
  for (int b = threadIdx.x; b < nbucket; b += kT) s_bucket[b] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (uint32_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const BoxDev &bx = boxes[tile_box(boxes, nbox, tile)];
    const IngestBox<PT> ib(bx);
    const uint64_t i = (uint64_t)(tile - bx.tile_base) * (kT * PER) + threadIdx.x * PER;
    PT x[PER][3];
    load_some<PT, PER>(bx, i, x);
    uint32_t sum = 0;  // kept << 16 | images (of 1024 particles at most 26 624)
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const uint32_t o = i + j < bx.n ? ib.opts(x[j]) : 0u;
      if (!o) continue;
      sum += 65536u + opt_records(o) - 1u;
      if (nbucket > 1) {
        const uint32_t layer = opt_count(o, 0) * opt_count(o, 1);
        atomicAdd(s_bucket + ib.bucket(x[j][2]), layer);
        if (o & 16u) atomicAdd(s_bucket + ib.bucket(image_coord<PT>(bx.g, x[j][2], 2, -1)), layer);
        if (o & 32u) atomicAdd(s_bucket + ib.bucket(image_coord<PT>(bx.g, x[j][2], 2, 1)), layer);
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
    if (lane == 0) s_warp[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t t = 0;
#pragma unroll
      for (int w = 0; w < kT / 32; w++) t += s_warp[w];
      tile_sum[tile] = make_uint2(t >> 16, t & 0xffffu);
    }
    __syncthreads();
  }
  for (int b = threadIdx.x; b < nbucket; b += kT)
    if (s_bucket[b]) atomicAdd(bucket_count + b, s_bucket[b]);
}

// One CTA: exclusive prefixes over the tiles (in place) and the buckets (their
// first places), and per box the kept and image counts and the first
// processing index (its kept particles, then its images).  Sets the run's
// processed count, clamped to the capacity `np_cap`.
constexpr int kScanT = 1024;

__device__ __forceinline__ uint2 block_exclusive2(uint2 v, uint2 *s_warp, uint2 *total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint2 inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, inc.x, d);
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc.y, d);
    if (lane >= d) inc.x += x, inc.y += y;
  }
  if (lane == 31) s_warp[w] = inc;
  __syncthreads();
  uint2 before = make_uint2(0u, 0u), all = before;
  for (int q = 0; q < kScanT / 32; q++) {
    const uint2 t = s_warp[q];
    if (q < w) before.x += t.x, before.y += t.y;
    all.x += t.x;
    all.y += t.y;
  }
  __syncthreads();
  *total = all;
  return make_uint2(before.x + inc.x - v.x, before.y + inc.y - v.y);
}

__global__ void __launch_bounds__(kScanT) k_ingest_scan(const BoxDev *__restrict__ boxes, int nbox,
                                                        uint32_t ntile, int nbucket,
                                                        uint2 *tile_sum, uint32_t *bucket,
                                                        DevScal *sc, uint32_t *boxd,
                                                        uint32_t np_cap) {
  // boxd layout: [kept_before | img_before | nkept | nimg | proc_base | halo_count | halo_base]
  __shared__ uint2 s_warp[kScanT / 32];
  __shared__ uint32_t s_edge[2][kMaxBoxes + 1];
  constexpr uint32_t kItems = 8;
  uint2 carry = make_uint2(0u, 0u);
  for (uint32_t t0 = 0; t0 < ntile; t0 += kScanT * kItems) {
    uint2 v[kItems], sum = make_uint2(0u, 0u);
#pragma unroll
    for (uint32_t q = 0; q < kItems; q++) {
      const uint32_t t = t0 + threadIdx.x * kItems + q;
      v[q] = t < ntile ? tile_sum[t] : make_uint2(0u, 0u);
      sum.x += v[q].x;
      sum.y += v[q].y;
    }
    uint2 total, run = block_exclusive2(sum, s_warp, &total);
    run.x += carry.x;
    run.y += carry.y;
#pragma unroll
    for (uint32_t q = 0; q < kItems; q++) {
      const uint32_t t = t0 + threadIdx.x * kItems + q;
      if (t < ntile) tile_sum[t] = run;
      run.x += v[q].x;
      run.y += v[q].y;
    }
    carry.x += total.x;
    carry.y += total.y;
  }
  __syncthreads();
  // the boxes' first tiles give what lies before each box (this CTA's writes)
  for (int b = threadIdx.x; b < nbox; b += kScanT) {
    const uint32_t t = boxes[b].tile_base;
    s_edge[0][b] = t < ntile ? tile_sum[t].x : carry.x;
    s_edge[1][b] = t < ntile ? tile_sum[t].y : carry.y;
  }
  if (threadIdx.x == 0) {
    s_edge[0][nbox] = carry.x;
    s_edge[1][nbox] = carry.y;
    const uint64_t np = (uint64_t)carry.x + carry.y;
    sc->kept_total = carry.x;
    sc->img_total = carry.y;
    sc->np_raw = np > 0xffffffffull ? 0xffffffffu : (uint32_t)np;
    sc->np = np > np_cap ? np_cap : (uint32_t)np;
    if (np > np_cap) atomicOr(&sc->overflow, 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nbox; b += kScanT) {
    const uint32_t k0 = s_edge[0][b], m0 = s_edge[1][b];
    boxd[0 * nbox + b] = k0;
    boxd[1 * nbox + b] = m0;
    boxd[2 * nbox + b] = s_edge[0][b + 1] - k0;
    boxd[3 * nbox + b] = s_edge[1][b + 1] - m0;
    boxd[4 * nbox + b] = k0 + m0;
  }
  uint32_t bcarry = 0;
  for (int b0 = 0; b0 < nbucket; b0 += kScanT) {
    const int b = b0 + (int)threadIdx.x;
    // (one bucket's counts are not taken: it holds everything)
    const uint32_t v = b < nbucket && nbucket > 1 ? bucket[b] : 0u;
    uint2 total;
    const uint2 ex = block_exclusive2(make_uint2(v, 0u), s_warp, &total);
    if (b < nbucket) bucket[b] = bcarry + ex.x;
    bcarry += total.x;
  }
}

// Fine-cell key of a processed particle at c: (top cell, counted over the
// run's boxes) * k^3 + the fine cell within it.  c holds the stored (PT)
// coordinates, so the fine cell can be recomputed from the stored position.
__device__ __forceinline__ uint64_t cell_key(const Geom &g, uint64_t top_base, uint64_t k3all,
                                             const double c[3]) {
  int gi[3];
#pragma unroll
  for (int a = 0; a < 3; a++) gi[a] = fine_index(c[a], g.rmin[a], g.inv_h, g.G[a]);
  const int k = g.k;
  const int t[3] = {div_k(gi[0], g), div_k(gi[1], g), div_k(gi[2], g)};
  const uint64_t top = top_base + ((uint64_t)t[2] * g.T[1] + t[1]) * g.T[0] + t[0];
  const uint64_t sub = ((uint64_t)(gi[2] - t[2] * k) * k + (gi[1] - t[1] * k)) * k + (gi[0] - t[0] * k);
  return top * k3all + sub;
}

// Writes a record (one 32-byte store for float positions).
__device__ __forceinline__ void store_rec(PRec<float> *to, const double c[3], uint32_t src,
                                          uint64_t key, uint32_t proc) {
  const uint64_t w0 = (uint64_t)__float_as_uint((float)c[0]) |
                      (uint64_t)__float_as_uint((float)c[1]) << 32;
  const uint64_t w1 = (uint64_t)__float_as_uint((float)c[2]) | (uint64_t)src << 32;
  asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(to), "l"(w0), "l"(w1), "l"(key),
               "l"((uint64_t)proc)
               : "memory");
}
__device__ __forceinline__ void store_rec(PRec<double> *to, const double c[3], uint32_t src,
                                          uint64_t key, uint32_t proc) {
  double2 *q = reinterpret_cast<double2 *>(to);
  q[0] = make_double2(c[0], c[1]);
  q[1] = make_double2(c[2], __longlong_as_double((long long)key));
  reinterpret_cast<uint4 *>(to)[2] = make_uint4(src, proc, 0u, 0u);
}

// Emission of the records of a tile into their buckets.  Each particle takes
// a run of places per layer of images (its own z, then z - L, z + L), counted
// in shared memory; the tile takes its places of each bucket with one atomic.
// Processing order of a box: kept originals in input order, then the images
// grouped by source particle and shift code (sz+1)*9 + (sy+1)*3 + (sx+1)
// ascending; the index is computed from the tile's prefixes.  The images are
// emitted one per thread, found by a search in the tile's image prefix, so
// that image work is proportional to the images.  Writes beyond the capacity
// are dropped (the run is then repeated with more room).  The records' digits
// for all passes of the sort are counted on the way.
template <class PT, int PER>
__global__ void __launch_bounds__(kT) k_ingest_emit(
    const BoxDev *__restrict__ boxes, int nbox, uint32_t ntile, int nbucket, uint64_t k3all,
    const uint2 *__restrict__ tile_sum, uint32_t *__restrict__ bucket,
    const uint32_t *__restrict__ boxd, uint32_t np_cap, PRec<PT> *__restrict__ recs,
    PassDigits pd, uint32_t *__restrict__ ghist) {
  extern __shared__ uint32_t s_hist[];        // the sort's digit counts of this CTA's records
  __shared__ uint32_t s_count[kMaxBuckets];   // records of the tile, then their first place
  __shared__ uint32_t s_warp[kT / 32];
  __shared__ uint32_t s_img[kT + 1];          // images before each thread's particles
  // per particle: opts | rank of its own layer << 16 | of z - L << 32 | of z + L << 48
  __shared__ uint64_t s_part[kT * PER];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int q = threadIdx.x; q < pd.passes * kRadixBins; q += kT) s_hist[q] = 0;
  auto put = [&](uint32_t at, const double (&c)[3], uint32_t src, uint64_t key, uint32_t proc) {
    if (at >= np_cap) return;
    store_rec(recs + at, c, src, key, proc);
#pragma unroll
    for (int q = 0; q < kRadixPasses; q++)
      if (q < pd.passes)
        atomicAdd(s_hist + q * kRadixBins +
                      ((uint32_t)(key >> pd.shift[q]) & ((1u << pd.width[q]) - 1u)), 1u);
  };
  for (uint32_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int b = tile_box(boxes, nbox, tile);
    const BoxDev &bx = boxes[b];
    const Geom &g = bx.g;
    const IngestBox<PT> ib(bx);
    // the tile touches its own box's buckets only
    const int b0 = (int)bx.bucket_base, b1 = b0 + (int)bx.nbucket;
    for (int q = b0 + (int)threadIdx.x; q < b1; q += kT) s_count[q] = 0;
    const uint64_t i = (uint64_t)(tile - bx.tile_base) * (kT * PER) + threadIdx.x * PER;
    PT x[PER][3];
    load_some<PT, PER>(bx, i, x);
    __syncthreads();
    uint32_t sum = 0, opts[PER], rank[PER], where[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const uint32_t o = i + j < bx.n ? ib.opts(x[j]) : 0u;
      opts[j] = o;
      rank[j] = where[j] = 0;
      uint64_t ranks = 0;
      if (o) {
        sum += 65536u + opt_records(o) - 1u;
        const uint32_t layer = opt_count(o, 0) * opt_count(o, 1);
        const PT z = x[j][2];
        where[j] = ib.bucket(z);
        rank[j] = atomicAdd(s_count + where[j], layer);
        ranks = (uint64_t)rank[j] << 16;
        if (o & 16u)
          ranks |= (uint64_t)atomicAdd(s_count + ib.bucket(image_coord<PT>(g, z, 2, -1)), layer)
                   << 32;
        if (o & 32u)
          ranks |= (uint64_t)atomicAdd(s_count + ib.bucket(image_coord<PT>(g, z, 2, 1)), layer)
                   << 48;
      }
      s_part[threadIdx.x * PER + j] = ranks | o;
    }
    // kept << 16 | images before this thread's particles
    uint32_t inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += t;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    uint32_t before = inc - sum, total = 0;
#pragma unroll
    for (int q = 0; q < kT / 32; q++) {
      if (q < w) before += s_warp[q];
      total += s_warp[q];
    }
    s_img[threadIdx.x] = before & 0xffffu;
    for (int q = b0 + (int)threadIdx.x; q < b1; q += kT)
      if (s_count[q]) s_count[q] = atomicAdd(bucket + q, s_count[q]);
    __syncthreads();
    const uint2 ts = tile_sum[tile];
    const uint32_t pbase = boxd[4 * nbox + b];
    uint32_t p = pbase + (ts.x - boxd[0 * nbox + b]) + (before >> 16);
#pragma unroll
    for (int j = 0; j < PER; j++) {
      if (!opts[j]) continue;
      const double c[3] = {as_d(x[j][0]), as_d(x[j][1]), as_d(x[j][2])};
      put(s_count[where[j]] + rank[j], c, (uint32_t)(bx.in_base + i + j),
          cell_key(g, bx.top_base, k3all, c), p);
      p++;
    }
    // the tile's images, one per thread: a particle's images are the product
    // of its per-axis options (-1 | 0 | +1 where the shifted coordinate stays
    // in the shell) without (0, 0, 0), in z, y, x order
    const uint32_t nimg = total & 0xffffu;
    const uint32_t qbase = pbase + boxd[2 * nbox + b] + (ts.y - boxd[1 * nbox + b]);
    for (uint32_t m = threadIdx.x; m < nimg; m += kT) {
      int lo = 0, hi = kT - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_img[mid] <= m) lo = mid;
        else hi = mid - 1;
      }
      uint32_t r = m - s_img[lo];
      int j = 0;
      uint64_t part = s_part[lo * PER];
      while (j < PER - 1) {
        const uint32_t ni = (part & 127u) ? opt_records((uint32_t)part & 127u) - 1u : 0u;
        if (r < ni) break;
        r -= ni;
        part = s_part[lo * PER + ++j];
      }
      const uint32_t o = (uint32_t)part & 127u;
      const int nx = (int)opt_count(o, 0), ny = (int)opt_count(o, 1);
      const int zx = (int)(o & 1u), zy = (int)((o >> 2) & 1u), zz = (int)((o >> 4) & 1u);
      const uint32_t own = (uint32_t)((zz * ny + zy) * nx + zx);  // (0, 0, 0) in that order
      const uint32_t e = r + (r >= own ? 1u : 0u);
      const int ex = (int)(e % (uint32_t)nx), ey = (int)((e / (uint32_t)nx) % (uint32_t)ny),
                ez = (int)(e / (uint32_t)(nx * ny));
      const int sh[3] = {ex - zx, ey - zy, ez - zz};
      const uint64_t li = (uint64_t)(tile - bx.tile_base) * (kT * PER) + (uint64_t)(lo * PER + j);
      double c[3];
      load_pos<PT>(bx, li, c);
#pragma unroll
      for (int a = 0; a < 3; a++)
        if (sh[a] != 0) c[a] = (double)image_coord<PT>(g, (PT)c[a], a, sh[a]);
      // its place in its layer: in the own layer the particle itself is first
      const uint32_t in_layer = (uint32_t)(ey * nx + ex), self = (uint32_t)(zy * nx + zx);
      const uint32_t rk = (uint32_t)(part >> (sh[2] == 0 ? 16 : sh[2] < 0 ? 32 : 48)) & 0xffffu;
      const uint32_t at = s_count[ib.bucket((PT)c[2])] + rk +
                          (sh[2] == 0 ? in_layer + (in_layer < self ? 1u : 0u) : in_layer);
      put(at, c, (uint32_t)(bx.in_base + li), cell_key(g, bx.top_base, k3all, c), qbase + m);
    }
    __syncthreads();
  }
  __syncthreads();
  for (int q = threadIdx.x; q < pd.passes * kRadixBins; q += kT)
    if (s_hist[q]) atomicAdd(ghist + q, s_hist[q]);
}

// ---------------------------------------------------------------------------
// Runs of equal fine-cell keys.
// ---------------------------------------------------------------------------

// Fine cell of a stored processed particle, packed gx | gy << 21 | gz << 42,
// and its box: the stored coordinates are those its sort key was computed
// from, so (box, fine cell) is that key's exactly.
template <class PT>
__device__ __forceinline__ uint64_t stored_cell(const BoxDev *boxes, const uint64_t *s_base,
                                                int nbox, const SPos<PT> &sp, int *box) {
  const int b = nbox > 1 ? box_search(s_base, nbox, (uint64_t)sp.src) : 0;
  const Geom &g = boxes[b].g;
  const double c[3] = {as_d(sp.x), as_d(sp.y), as_d(sp.z)};
  uint64_t packed = 0;
#pragma unroll
  for (int a = 0; a < 3; a++)
    packed |= (uint64_t)fine_index(c[a], g.rmin[a], g.inv_h, g.G[a]) << (21 * a);
  *box = b;
  return packed;
}

// Reads a record (one 32-byte load for float positions).
__device__ __forceinline__ void load_rec(const PRec<float> *from, SPos<float> *p, uint32_t *proc) {
  uint64_t w0, w1, key, tail;
  asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
               : "=l"(w0), "=l"(w1), "=l"(key), "=l"(tail)
               : "l"(from));
  p->x = __uint_as_float((uint32_t)w0);
  p->y = __uint_as_float((uint32_t)(w0 >> 32));
  p->z = __uint_as_float((uint32_t)w1);
  p->src = (uint32_t)(w1 >> 32);
  *proc = (uint32_t)tail;
}
__device__ __forceinline__ void load_rec(const PRec<double> *from, SPos<double> *p,
                                         uint32_t *proc) {
  const double2 a = reinterpret_cast<const double2 *>(from)[0];
  p->x = a.x;
  p->y = a.y;
  p->z = from->z;
  const uint4 t = reinterpret_cast<const uint4 *>(from)[2];
  p->src = t.x;
  p->pad = 0;
  *proc = t.y;
}

__device__ __forceinline__ uint64_t top_of_run(const BoxDev &bx, uint64_t pg) {
  const Geom &g = bx.g;
  const int gx = (int)(pg & kM21), gy = (int)((pg >> 21) & kM21), gz = (int)(pg >> 42);
  return bx.top_base +
         ((uint64_t)div_k(gz, g) * g.T[1] + (uint64_t)div_k(gy, g)) * g.T[0] + div_k(gx, g);
}

// Tile states of the run count's look-back, as the sort's: the flag in the high
// half, the count in the low half.
constexpr uint64_t kTileOwn = 1ull << 32;   // the tile's own runs
constexpr uint64_t kTileAll = 2ull << 32;   // the runs up to and with this tile

// Runs before `tile`: one warp adds up the lower tiles' published states, 32 at
// a time, back to the first inclusive one.  Every lower tile publishes its own
// count before it waits, so every wait ends; a wait is capped all the same
// (`polls` reads) and then raises *failed and gives kNone.
__device__ __forceinline__ uint32_t runs_before(const uint64_t *state, uint32_t tile,
                                                uint32_t polls, unsigned int *failed) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t sum = 0, left = polls;
  int64_t top = (int64_t)tile - 1;
  while (top >= 0) {
    const int64_t j = top - (int64_t)lane;
    uint64_t w = kTileAll;  // (below tile 0: nothing)
    if (j >= 0) w = *reinterpret_cast<const volatile uint64_t *>(state + j);
    const uint32_t all = __ballot_sync(0xffffffffu, (w >> 32) == 2);
    const uint32_t none = __ballot_sync(0xffffffffu, (w >> 32) == 0);
    const int first = all ? __ffs(all) - 1 : 31;  // the nearest inclusive state
    const uint32_t need = first == 31 ? 0xffffffffu : (2u << first) - 1u;
    if (none & need) {
      if (left-- == 0) {
        if (lane == 0) atomicAdd(failed, 1u);
        return kNone;
      }
      continue;
    }
    sum += __reduce_add_sync(0xffffffffu, (need >> lane) & 1u ? (uint32_t)w : 0u);
    if (all) break;
    top -= 32;
    left = polls;
  }
  return sum;
}

// The records in cell order and their runs (of equal box and fine cell), in one
// sweep: positions, processing indices and runs of the particles; per run its
// first particle, packed fine cell (the sort leaves only the order: it is
// recomputed), box and initial parent (itself); the range of runs of every
// occupied top cell (top_range starts zeroed; where the top cell changes
// between two particles, the new one's first run is the old one's end).  A tile
// counts its run starts, publishes the count and learns the lower tiles' by
// look-back; one that gives up writes no runs.  The failed flag may be raised
// while this kernel runs, so one thread reads it for its whole CTA, before it
// takes a tile (the tiles taken are all worked on).  A gather, a three-kernel
// scan of start flags and a kernel for the runs moved 40 bytes more per particle:
// 0.60 ms on the 256^3 box, this 0.37; 512^3 box 5.9 and 2.9 ms.
//
// A warp has 32 PER consecutive elements, 32 at a time; lane l compares with lane
// l - 1's cell, lane 0 with the last of the 32 before (before the first 32 it
// recomputes its predecessor's).
// PER is 8 in large runs, where a tile's barriers and its wait for the lower
// tiles weigh more than the tiles' number (512^3 box 3.33 ms with 4, 3.09 with 8,
// 3.51 with 16), and 4 in small ones (10,007 particles: 16 and 18 us).
constexpr int kRunPerSmall = 4, kRunPerLarge = 8;

template <class PT, int kRunPer>
__global__ void __launch_bounds__(kT) k_gather_runs(
    const uint32_t *__restrict__ order, const PRec<PT> *__restrict__ recs,
    const BoxDev *__restrict__ boxes, int nbox, SPos<PT> *__restrict__ spos,
    uint32_t *__restrict__ perm, uint32_t *__restrict__ run_of, uint32_t *__restrict__ run_start,
    uint64_t *__restrict__ run_g, uint16_t *__restrict__ run_box, uint32_t *__restrict__ parent,
    uint32_t *__restrict__ top_range, uint64_t *state, DevScal *sc, SortWaits waits) {
  constexpr int kRunTile = kT * kRunPer;
  __shared__ uint64_t s_base[kMaxBoxes];
  __shared__ uint32_t s_tile, s_warp[kT / 32], s_before;
  if (threadIdx.x == 0)  // (after a sort that gave up the order is not valid)
    s_tile = __ldcg(&sc->failed) ? kNone : atomicAdd(&sc->next_tile, 1u);
  load_bases(boxes, nbox, s_base, false);
  const uint32_t tile = s_tile;
  const int64_t np = sc->np;
  if (tile == kNone || (int64_t)tile * kRunTile >= np) return;  // the whole CTA leaves together
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)tile * kRunTile + w * (32 * kRunPer) + lane;
  uint32_t from[kRunPer], before = 0;
#pragma unroll
  for (int j = 0; j < kRunPer; j++) from[j] = i0 + 32 * j < np ? order[i0 + 32 * j] : 0u;
  const bool has_before = lane == 0 && i0 > 0 && i0 < np;
  if (has_before) before = order[i0 - 1];
  SPos<PT> sp[kRunPer], sq;
  uint32_t proc[kRunPer], unused;
#pragma unroll
  for (int j = 0; j < kRunPer; j++)
    if (i0 + 32 * j < np) load_rec(recs + from[j], &sp[j], &proc[j]);
  if (has_before) load_rec(recs + before, &sq, &unused);
  uint64_t cell[kRunPer], pcell[kRunPer];
  int box[kRunPer], pbox[kRunPer];
  uint32_t start[kRunPer];  // the warp's run starts
  uint64_t last_cell = 0;
  int last_box = 0;
  if (has_before) last_cell = stored_cell<PT>(boxes, s_base, nbox, sq, &last_box);
#pragma unroll
  for (int j = 0; j < kRunPer; j++) {
    const int64_t i = i0 + 32 * j;
    cell[j] = 0;
    box[j] = 0;
    if (i < np) {
      spos[i] = sp[j];
      perm[i] = proc[j];
      cell[j] = stored_cell<PT>(boxes, s_base, nbox, sp[j], &box[j]);
    }
    pcell[j] = __shfl_up_sync(0xffffffffu, cell[j], 1);
    pbox[j] = __shfl_up_sync(0xffffffffu, box[j], 1);
    if (lane == 0) {
      pcell[j] = last_cell;
      pbox[j] = last_box;
    }
    last_cell = __shfl_sync(0xffffffffu, cell[j], 31);
    last_box = __shfl_sync(0xffffffffu, box[j], 31);
    start[j] = __ballot_sync(0xffffffffu,
                             i < np && (i == 0 || cell[j] != pcell[j] || box[j] != pbox[j]));
  }
  uint32_t mine = 0;
#pragma unroll
  for (int j = 0; j < kRunPer; j++) mine += __popc(start[j]);
  if (lane == 0) s_warp[w] = mine;
  __syncthreads();
  uint32_t in_tile = 0, wbefore = 0;
#pragma unroll
  for (uint32_t q = 0; q < kT / 32; q++) {
    if (q < w) wbefore += s_warp[q];
    in_tile += s_warp[q];
  }
  if (w == 0) {
    unsigned long long *own = reinterpret_cast<unsigned long long *>(state + tile);
    // (a tile named by waits.stall_tile publishes nothing: a test hook whose
    // successor's capped wait then runs out)
    const bool publish = lane == 0 && tile != waits.stall_tile;
    if (publish && tile != 0) atomicExch(own, (unsigned long long)(kTileOwn | in_tile));
    const uint32_t b = runs_before(state, tile, waits.spin_cap, &sc->failed);
    // (after a give-up any count in range will do: the next tiles' waits end)
    if (publish) atomicExch(own, (unsigned long long)(kTileAll | ((b == kNone ? 0u : b) + in_tile)));
    if (lane == 0) s_before = b;
  }
  __syncthreads();
  if (s_before == kNone) return;
  uint32_t done = s_before + wbefore;  // runs that start before these 32
#pragma unroll
  for (int j = 0; j < kRunPer; j++) {
    const int64_t i = i0 + 32 * j;
    const uint32_t rid = done + __popc(start[j] & ((2u << lane) - 1u)) - 1u;
    done += __popc(start[j]);
    if (i >= np) continue;
    run_of[i] = rid;
    if (!((start[j] >> lane) & 1u) && i != np - 1) continue;
    const uint64_t t = top_of_run(boxes[box[j]], cell[j]);
    if ((start[j] >> lane) & 1u) {
      run_start[rid] = (uint32_t)i;
      run_g[rid] = cell[j];
      run_box[rid] = (uint16_t)box[j];
      parent[rid] = rid;
      const uint64_t pt = i > 0 ? top_of_run(boxes[pbox[j]], pcell[j]) : t;
      if (i == 0 || pt != t) top_range[2 * t] = rid;
      if (pt != t) top_range[2 * pt + 1] = rid;
    }
    if (i == np - 1) {
      top_range[2 * t + 1] = rid + 1u;
      run_start[rid + 1u] = (uint32_t)np;
      sc->R = rid + 1u;
    }
  }
}

// Grid cell and linking length of every processed particle (variable
// linking length runs only; boxes with a fixed length get cell 0 and their
// own l^2, which reproduces the fixed-length test).
template <class PT, bool FP32>
__global__ void __launch_bounds__(kT) k_varlink_recs(const SPos<PT> *__restrict__ spos,
                                                     const uint32_t *__restrict__ run_of,
                                                     const uint16_t *__restrict__ run_box,
                                                     const BoxDev *__restrict__ boxes,
                                                     const DevScal *__restrict__ sc,
                                                     VLRec<FP32> *__restrict__ svl) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const int64_t np = sc->np;
  for (int64_t i = gtid(); i < np; i += gstride()) {
    const Geom &g = boxes[run_box[run_of[i]]].g;
    VLRec<FP32> v;
    v.rkey = 0;
    v.lsq = g.linksq;
    if (g.varlink) {
      const SPos<PT> p = spos[i];
      v.rkey = ref_key(g, (double)p.x, (double)p.y, (double)p.z);
      v.lsq = ref_cell_linksq(g, v.rkey);
    }
    svl[i] = v;
  }
}

// Warp-aggregated slot from a counter for the lanes with `pick` set: one
// atomic per warp, the lanes in lane order after the returned base.
__device__ __forceinline__ uint32_t warp_slot(bool pick, uint32_t *counter) {
  const uint32_t m = __ballot_sync(0xffffffffu, pick);
  if (m == 0) return 0u;
  const int lane = threadIdx.x & 31, first = __ffs(m) - 1;
  uint32_t base = 0;
  if (lane == first) base = atomicAdd(counter, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, first);
  return base + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// Dense top cells (more than dense_min fine cells), one thread per fine
// cell, acting at each top cell's first: a slot from a counter (the order of
// the slots does not matter), the top cell's slot and fine-cell range, and
// the big ones' slots listed in `big`.  Past nd_cap a dense top cell gets no
// slot and is scanned instead (slower but exact), and the overflow bit asks
// the plan for more slots next time.
__global__ void __launch_bounds__(kT) k_dense_pick(const uint64_t *__restrict__ run_g,
                                                   const uint16_t *__restrict__ run_box,
                                                   const BoxDev *__restrict__ boxes,
                                                   DevScal *sc,
                                                   const uint2 *__restrict__ top_range,
                                                   uint32_t dense_min, uint32_t big_min,
                                                   uint32_t nd_cap,
                                                   uint32_t *__restrict__ top_slot,
                                                   uint2 *__restrict__ dense_range,
                                                   uint32_t *__restrict__ big) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const uint32_t R = sc->R;
  const int lane = threadIdx.x & 31;
  for (int64_t r0 = gtid() - lane; r0 < (int64_t)R; r0 += gstride()) {
    const int64_t r = r0 + lane;
    bool pick = false;
    uint64_t t = 0;
    uint2 tr = make_uint2(0u, 0u);
    if (r < (int64_t)R) {
      t = top_of_run(boxes[run_box[r]], run_g[r]);
      tr = top_range[t];
      pick = tr.x == (uint32_t)r && tr.y - tr.x > dense_min;
    }
    const uint32_t slot = warp_slot(pick, &sc->nd);
    if (!pick) continue;
    if (slot < nd_cap) {
      top_slot[t] = slot;
      dense_range[slot] = tr;
      if (tr.y - tr.x > big_min) big[atomicAdd(&sc->nbig, 1u)] = slot;
    } else {
      atomicOr(&sc->overflow, 2u);
    }
  }
}


// ---------------------------------------------------------------------------
// Befriending.
// ---------------------------------------------------------------------------

// The reference's pair predicate (FOF.c:351-357), FP64 or FP32 + band recheck.
// With VL (variable linking length) the pair's l^2 or band comes from the
// lower of the two particles' grid cells, and particles of cells that are
// not neighbours are never linked; va/vb are ignored otherwise.
template <class PT, bool FP32, bool VL>
__device__ __forceinline__ bool linked(const SPos<PT> &p, const SPos<PT> &q, const Geom &g,
                                       const VLRec<FP32> &va, const VLRec<FP32> &vb,
                                       uint32_t &rechecks) {
  float t_lo = g.t_lo, t_hi = g.t_hi;
  double lsq = g.linksq;
  if constexpr (VL) {
    if (!ref_neighbours(va.rkey, vb.rkey)) return false;
    lsq = (va.rkey <= vb.rkey ? va : vb).lsq;
    if constexpr (FP32) vl_band(lsq, sizeof(PT) == 4 ? 4 : 8, &t_lo, &t_hi);
  }
  double dx, dy, dz;
  if constexpr (sizeof(PT) == 4) {
    const float fx = __fsub_rn(p.x, q.x), fy = __fsub_rn(p.y, q.y), fz = __fsub_rn(p.z, q.z);
    if constexpr (FP32) {
      const float d2 = __fmaf_rn(fz, fz, __fmaf_rn(fy, fy, __fmul_rn(fx, fx)));
      if (d2 < t_lo) return true;
      if (d2 > t_hi) return false;
      rechecks++;
    }
    dx = (double)fx;
    dy = (double)fy;
    dz = (double)fz;
  } else {
    dx = __dsub_rn(p.x, q.x);
    dy = __dsub_rn(p.y, q.y);
    dz = __dsub_rn(p.z, q.z);
    if constexpr (FP32) {
      const float fx = __double2float_rn(dx), fy = __double2float_rn(dy),
                  fz = __double2float_rn(dz);
      const float d2 = __fmaf_rn(fz, fz, __fmaf_rn(fy, fy, __fmul_rn(fx, fx)));
      if (d2 < t_lo) return true;
      if (d2 > t_hi) return false;
      rechecks++;
    }
  }
  const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return !(d2 > lsq);
}

// Squared distance from a point to the box of fine cell (cx, cy, cz).
__device__ __forceinline__ double box_dist2(const Geom &g, double x, double y, double z, int cx,
                                            int cy, int cz) {
  const double bx = __dadd_rn(g.rmin[0], __dmul_rn((double)cx, g.h));
  const double by = __dadd_rn(g.rmin[1], __dmul_rn((double)cy, g.h));
  const double bz = __dadd_rn(g.rmin[2], __dmul_rn((double)cz, g.h));
  const double ex = fmax(0.0, fmax(bx - x, x - (bx + g.h)));
  const double ey = fmax(0.0, fmax(by - y, y - (by + g.h)));
  const double ez = fmax(0.0, fmax(bz - z, z - (bz + g.h)));
  return ex * ex + ey * ey + ez * ez;
}

// Per-thread tallies of the befriending kernels, flushed once per warp.  They are
// 32 bits wide (registers): spill() moves them to the counters before they
// wrap, between the kernels' items, none of which adds 2^31, and between the
// steps of a search of two crowded cells, which can take any number.
struct BfStats {
  uint32_t tests = 0, rechecks = 0, cand = 0, skips = 0, unions = 0, steps = 0;
  uint32_t scan = 0, window = 0;

  // (by any lane for itself)
  __device__ __forceinline__ void spill(Counters *ctr) {
    if (!((tests | rechecks | cand | skips | unions | steps | scan | window) >> 31)) return;
    auto move = [](unsigned long long *to, uint32_t &v) {
      if (v) atomicAdd(to, (unsigned long long)v);
      v = 0;
    };
    move(&ctr->pair_tests, tests);
    move(&ctr->rechecks, rechecks);
    move(&ctr->cand_pairs, cand);
    move(&ctr->root_skips, skips);
    move(&ctr->unions, unions);
    move(&ctr->find_steps, steps);
    move(&ctr->scan_iters, scan);
    move(&ctr->window_iters, window);
  }
  __device__ void add(unsigned long long *to, uint32_t v) {
    unsigned long long w = v;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) w += __shfl_down_sync(0xffffffffu, w, d);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(to, w);
  }
  __device__ void flush(Counters *ctr) {
    add(&ctr->pair_tests, tests);
    add(&ctr->rechecks, rechecks);
    add(&ctr->cand_pairs, cand);
    add(&ctr->root_skips, skips);
    add(&ctr->unions, unions);
    add(&ctr->find_steps, steps);
    add(&ctr->scan_iters, scan);
    add(&ctr->window_iters, window);
  }
};

// Whether any particle of fine cell a (particles [sa, ea), packed fine
// coordinates ga) is linked to any particle of fine cell b ([sb, eb), gb):
// 1 or 0, or 2 when `limit` steps did not tell.
// The loop runs over the cell with fewer particles, and each of its
// particles farther than the linking length from the other cell's box is
// skipped; the pair predicate is symmetric (the difference of a pair
// only changes sign, and a variable length comes from the lower of the two
// grid cells), so the orientation does not change the answer.
template <class PT, bool FP32, bool VL>
__device__ __forceinline__ int cells_linked(const Geom &g, uint64_t ga, uint64_t gb, uint32_t sa,
                                            uint32_t ea, uint32_t sb, uint32_t eb, int limit,
                                            const SPos<PT> *__restrict__ spos,
                                            const VLRec<FP32> *__restrict__ svl, BfStats &st) {
  if (eb - sb < ea - sa) {
    uint32_t t = sa;
    sa = sb;
    sb = t;
    t = ea;
    ea = eb;
    eb = t;
    gb = ga;
  }
  const int bx = (int)(gb & kM21), by = (int)((gb >> 21) & kM21), bz = (int)(gb >> 42);
  for (uint32_t i = sa; i < ea; i++) {
    const SPos<PT> p = spos[i];
    if (limit-- <= 0) return 2;
    if (box_dist2(g, (double)p.x, (double)p.y, (double)p.z, bx, by, bz) > g.prune_sq) continue;
    VLRec<FP32> va{};
    if constexpr (VL) va = svl[i];
    for (uint32_t j = sb; j < eb; j++) {
      if (limit-- <= 0) return 2;
      st.tests++;
      VLRec<FP32> vb{};
      if constexpr (VL) vb = svl[j];
      if (linked<PT, FP32, VL>(p, spos[j], g, va, vb, st.rechecks)) return 1;
    }
  }
  return 0;
}

// Union-find in shared memory over the fine cells of one top cell (local
// indices), same hook-to-min rule as the global one.
__device__ __forceinline__ uint32_t lfind(volatile uint32_t *lp, uint32_t x) {
  while (true) {
    const uint32_t p = lp[x];
    if (p == x) return x;
    const uint32_t gp = lp[p];
    if (gp == p) return p;
    lp[x] = gp;
    x = gp;
  }
}

// Returns whether this call joined two components.
__device__ __forceinline__ bool lunion(uint32_t *lp, uint32_t a, uint32_t b, Counters *ctr,
                                       uint32_t cap) {
  for (uint32_t it = 0; it < cap; it++) {
    a = lfind(lp, a);
    b = lfind(lp, b);
    if (a == b) return false;
    if (a < b) {
      const uint32_t t = a;
      a = b;
      b = t;
    }
    const uint32_t old = atomicCAS(lp + a, a, b);
    if (old == a) return true;
    a = old;
  }
  atomicAdd(&ctr->uf_giveups, 1u);
  return false;
}

// Bits lo..hi (0 <= lo <= hi <= 31) set.
__device__ __forceinline__ uint32_t bit_span(int lo, int hi) {
  return (hi - lo == 31 ? 0xffffffffu : ((1u << (hi - lo + 1)) - 1u)) << lo;
}

// The global union-find, and the one of a top cell's fine cells in shared
// memory (indices counted from the top cell's first fine cell, `first`).
struct GlobalUF {
  uint32_t *parent;
  __device__ __forceinline__ uint32_t find(uint32_t x, BfStats &st) const {
    return uf_find_n(parent, x, st.steps);
  }
  __device__ __forceinline__ void join(uint32_t a, uint32_t b, Counters *ctr, uint32_t cap) const {
    uf_union(parent, a, b, ctr, cap);
  }
};
struct LocalUF {
  uint32_t *lpar, *ncomp;
  uint32_t first;
  __device__ __forceinline__ uint32_t find(uint32_t x, BfStats &) const {
    return lfind(lpar, x - first);
  }
  __device__ __forceinline__ void join(uint32_t a, uint32_t b, Counters *ctr, uint32_t cap) const {
    if (lunion(lpar, a, b, ctr, cap)) atomicSub(ncomp, 1u);
  }
};

// Cell pairs a warp has found to be in reach and in different components,
// waiting to be tested: fewer than 32 are left over when 32 more may be added.
constexpr uint32_t kPairSlots = 64;
// Steps that one lane spends on a cell pair by itself; the whole warp takes
// those that need more, 32 particle pairs a step.  Most pairs that link do so
// within a few steps: 8, 16, 24 and 48 steps give a befriending of 1.09, 1.10,
// 1.11 and 1.13 ms for the 256^3 box and 0.154, 0.144, 0.149 and 0.158 ms for the
// 64^3 one; giving the warp every pair of more than 32 particle pairs made the
// dense kernel 1.6 times as long.
constexpr int kSoloSteps = 16;

// What the pair tests read, the same for all warps of a kernel.
template <class PT, bool FP32>
struct PairArgs {
  const BoxDev *boxes;
  const uint16_t *run_box;
  const uint32_t *run_start;
  const uint64_t *run_g;
  const SPos<PT> *spos;
  const VLRec<FP32> *svl;
  Counters *ctr;
};

// cells_linked() by a whole warp (same arguments on every lane): the lanes
// take 32 particles of the smaller cell at a time, drop those farther than
// the linking length from the other cell's box, and hold each one left
// against 32 particles of the other cell a step.  A search that one lane
// would run for thousands of dependent steps takes 1/32 of them.
template <class PT, bool FP32, bool VL, class UF>
__device__ __forceinline__ bool warp_cells_linked(const PairArgs<PT, FP32> &A, const UF &uf,
                                                  const Geom &g, uint64_t ga, uint64_t gb,
                                                  uint32_t a, uint32_t b, uint32_t sa,
                                                  uint32_t ea, uint32_t sb, uint32_t eb,
                                                  BfStats &st) {
  const uint32_t lane = threadIdx.x & 31;
  if (eb - sb < ea - sa) {
    uint32_t t = sa;
    sa = sb;
    sb = t;
    t = ea;
    ea = eb;
    eb = t;
    gb = ga;
  }
  const int bx = (int)(gb & kM21), by = (int)((gb >> 21) & kM21), bz = (int)(gb >> 42);
  for (uint32_t i0 = sa; i0 < ea; i0 += 32) {
    SPos<PT> p{};
    VLRec<FP32> va{};
    bool near = false;
    if (i0 + lane < ea) {
      p = A.spos[i0 + lane];
      near = !(box_dist2(g, (double)p.x, (double)p.y, (double)p.z, bx, by, bz) > g.prune_sq);
      if constexpr (VL) va = A.svl[i0 + lane];
    }
    uint32_t left = __ballot_sync(0xffffffffu, near);
    for (uint32_t step = 1; left; step++) {
      const int l = __ffs(left) - 1;
      left &= left - 1u;
      SPos<PT> q{};
      q.x = __shfl_sync(0xffffffffu, p.x, l);
      q.y = __shfl_sync(0xffffffffu, p.y, l);
      q.z = __shfl_sync(0xffffffffu, p.z, l);
      VLRec<FP32> vq{};
      if constexpr (VL) {
        vq.rkey = __shfl_sync(0xffffffffu, va.rkey, l);
        vq.lsq = __shfl_sync(0xffffffffu, va.lsq, l);
      }
      for (uint32_t j0 = sb; j0 < eb; j0 += 32) {
        const uint32_t j = j0 + lane;
        bool hit = false;
        if (j < eb) {
          VLRec<FP32> vb{};
          if constexpr (VL) vb = A.svl[j];
          st.tests++;
          hit = linked<PT, FP32, VL>(q, A.spos[j], g, vq, vb, st.rechecks);
        }
        if (__any_sync(0xffffffffu, hit)) return true;
      }
      st.spill(A.ctr);
      // joined by another warp meanwhile: the answer no longer matters
      if ((step & 7) == 0 && __any_sync(0xffffffffu, uf.find(a, st) == uf.find(b, st)))
        return false;
    }
  }
  return false;
}

// Tests the cell pairs in pairs[0, n), n <= 32, one per lane, and joins the
// linked ones: first whether the two cells are in one component by now, then
// a bounded number of tests by each lane, then the pairs that these did not
// settle one after another by the whole warp.
template <class PT, bool FP32, bool VL, class UF>
__device__ __forceinline__ void drain_pairs(const PairArgs<PT, FP32> &A, const UF &uf,
                                            const uint2 *pairs, uint32_t n, BfStats &st) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t a = 0, b = 0, sa = 0, ea = 0, sb = 0, eb = 0;
  uint64_t ga = 0, gb = 0;
  bool want = lane < n, big = false;
  if (want) {
    const uint2 pr = pairs[lane];
    a = pr.x;
    b = pr.y;
    sa = A.run_start[a];
    ea = A.run_start[a + 1];
    sb = A.run_start[b];
    eb = A.run_start[b + 1];
    ga = A.run_g[a];
    gb = A.run_g[b];
    const uint32_t ra = uf.find(a, st), rb = uf.find(b, st);
    want = ra != rb;
    if (!want) st.skips++;
    if (want) {
      const Geom &g = A.boxes[A.run_box[a]].g;
      const int is = cells_linked<PT, FP32, VL>(g, ga, gb, sa, ea, sb, eb, kSoloSteps, A.spos,
                                                A.svl, st);
      if (is == 1) {
        uf.join(ra, rb, A.ctr, g.union_cap);
        st.unions++;
      }
      big = is == 2;
    }
  }
  uint32_t todo = __ballot_sync(0xffffffffu, big);
  while (todo) {
    const int l = __ffs(todo) - 1;
    todo &= todo - 1u;
    const uint32_t la = __shfl_sync(0xffffffffu, a, l), lb = __shfl_sync(0xffffffffu, b, l);
    const uint32_t lsa = __shfl_sync(0xffffffffu, sa, l), lea = __shfl_sync(0xffffffffu, ea, l);
    const uint32_t lsb = __shfl_sync(0xffffffffu, sb, l), leb = __shfl_sync(0xffffffffu, eb, l);
    const uint64_t lga = __shfl_sync(0xffffffffu, ga, l), lgb = __shfl_sync(0xffffffffu, gb, l);
    const uint32_t ra = uf.find(la, st), rb = uf.find(lb, st);
    // (each lane looks for itself: the pair is skipped when any lane finds it joined)
    if (__any_sync(0xffffffffu, ra == rb)) {
      if ((int)lane == l) st.skips++;
      continue;
    }
    const Geom &g = A.boxes[A.run_box[la]].g;
    if (warp_cells_linked<PT, FP32, VL>(A, uf, g, lga, lgb, la, lb, lsa, lea, lsb, leb, st)) {
      if ((int)lane == l) {
        uf.join(ra, rb, A.ctr, g.union_cap);
        st.unions++;
      }
      __syncwarp();
    }
  }
}

// Adds the lanes' pairs (where `add` is set) to the warp's list and tests 32
// of them whenever it holds that many (with `last`, what it holds).  Called by
// all lanes, with fewer than 32 pairs in the list.
template <class PT, bool FP32, bool VL, class UF>
__device__ __forceinline__ void push_pairs(const PairArgs<PT, FP32> &A, const UF &uf, uint2 *pairs,
                                           uint32_t &npair, bool add, uint32_t a, uint32_t b,
                                           bool last, BfStats &st) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t m = __ballot_sync(0xffffffffu, add);
  if (add) pairs[npair + __popc(m & ((1u << lane) - 1u))] = make_uint2(a, b);
  npair += __popc(m);
  while (npair >= 32 || (last && npair)) {
    __syncwarp();
    const uint32_t n = min(npair, 32u);
    npair -= n;
    drain_pairs<PT, FP32, VL>(A, uf, pairs + npair, n, st);
    __syncwarp();
  }
}

// 16-byte words before the rows of a dense top cell's occupancy (2 k plane
// words and a fine cell's index).
__host__ __device__ constexpr int row_head(int k) { return (2 * k + 1 + 3) / 4; }

// Dense top cells: the fine-cell pairs inside a top cell are joined with a
// union-find in shared memory, near pairs before far ones; then every fine
// cell is joined to its local root in the global union-find (a
// compare-and-swap of its own parent when nothing else has hooked it, a
// union otherwise: the sparse kernel runs at the same time).  Links that cross the top
// cell's faces are left to the global passes.  The occupied fine cells of
// the top cell are first marked in bit rows (bit x of rows[z k + y]), so a
// cell visits only the occupied cells of its forward window, a row at a
// time, and finds their local indices from the rows' prefix counts.  A CTA shares the
// top cell when `cta` is set, else one warp has it; `lpar` holds
// k3all parents followed by the k^2 rows, their k^2 prefix counts, k^2 rows of
// the cells outside the main component and two single words; `pairs`
// is the warp's list of pairs to test.
template <class PT, bool FP32, bool VL>
__device__ __forceinline__ void dense_top(const PairArgs<PT, FP32> &A, uint32_t slot,
                                          uint32_t *lpar, bool cta, uint2 *pairs, uint64_t k3all,
                                          const uint2 *dense_range, uint4 *grows, uint32_t kk,
                                          uint32_t rows_stride, uint32_t *parent, BfStats &st) {
  const uint32_t tid = cta ? threadIdx.x : threadIdx.x & 31, nt = cta ? blockDim.x : 32;
  auto sync = [&]() {
    if (cta) __syncthreads();
    else __syncwarp();
  };
  const uint2 fr = dense_range[slot];
  const uint32_t f = fr.x, n = fr.y - fr.x;
  const Geom &g = A.boxes[A.run_box[f]].g;
  const int k = g.k, W = g.W;
  const uint32_t nrow = (uint32_t)(k * k);
  uint32_t *rows = lpar + k3all;   // occupancy bits of each (z, y) row
  uint32_t *pref = rows + nrow;    // occupied fine cells before each row
  uint32_t *rest = pref + nrow;    // the occupied fine cells outside the main component
  // components left: once one is left, every remaining candidate is joined
  volatile uint32_t *ncomp = lpar + k3all + 3 * kk, *vmain = ncomp + 1;
  const LocalUF uf{lpar, lpar + k3all + 3 * kk, f};
  if (tid == 0) *ncomp = n;
  for (uint32_t i = tid; i < n; i += nt) lpar[i] = i;
  for (uint32_t j = tid; j < nrow; j += nt) rows[j] = 0u;
  sync();
  for (uint32_t i = tid; i < n; i += nt) {
    const uint64_t pg = A.run_g[f + i];
    const int gx = (int)(pg & kM21), gy = (int)((pg >> 21) & kM21), gz = (int)(pg >> 42);
    atomicOr(rows + (gz - div_k(gz, g) * k) * k + (gy - div_k(gy, g) * k),
             1u << (gx - div_k(gx, g) * k));
  }
  sync();
  if (tid < 32) {
    // the top cell's fine cells are in sub-cell order, so a cell's local
    // index is the number of occupied cells in the rows before it plus those
    // before it in its row: prefix of the row populations, one warp
    const uint32_t per = (nrow + 31) / 32, j0 = tid * per, j1 = min(j0 + per, nrow);
    uint32_t sum = 0;
    for (uint32_t j = j0; j < j1; j++) sum += __popc(rows[j]);
    uint32_t inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
      if (tid >= (uint32_t)d) inc += t;
    }
    uint32_t acc = inc - sum;
    for (uint32_t j = j0; j < j1; j++) {
      pref[j] = acc;
      acc += __popc(rows[j]);
    }
  }
  sync();
  // The main component: the commonest root among 32 fine cells spread over the
  // top cell.  Most of the fine cells of a clump are in it once the near pairs
  // are joined, and for a cell of the main component only those in `rest` are
  // candidates still.
  auto find_main = [&]() {
    if (tid < 32) {
      const uint32_t r = lfind(lpar, (uint32_t)(((uint64_t)tid * n) >> 5));
      const uint32_t same = (uint32_t)__popc(__match_any_sync(0xffffffffu, r));
      const uint32_t most = __reduce_max_sync(0xffffffffu, same);
      const uint32_t who = __ballot_sync(0xffffffffu, same == most);
      const uint32_t m = __shfl_sync(0xffffffffu, r, __ffs(who) - 1);
      if (tid == 0) *vmain = m;
    }
    for (uint32_t j = tid; j < nrow; j += nt) rest[j] = 0u;
    sync();
    const uint32_t m = *vmain;
    for (uint32_t i = tid; i < n; i += nt) {
      if (lfind(lpar, i) == m) continue;
      const uint64_t pg = A.run_g[f + i];
      const int gx = (int)(pg & kM21), gy = (int)((pg >> 21) & kM21), gz = (int)(pg >> 42);
      atomicOr(rest + (gz - div_k(gz, g) * k) * k + (gy - div_k(gy, g) * k),
               1u << (gx - div_k(gx, g) * k));
    }
    sync();
  };
  uint32_t npair = 0;
  for (int pass = 0; pass < 3; pass++) {
    // pass 0: cells that share a face; pass 1: the others at Chebyshev distance
    // 1; pass 2: those at 2 and more.  Inside a clump the faces join nearly
    // everything, which leaves the other passes little to test.
    const int Wp = pass == 2 ? W : 1;
    if (pass >= 1) find_main();
    for (uint32_t i0 = tid & ~31u;; i0 += nt) {
      // past the warp's cells (or once one component is left; one answer for
      // the whole warp) the pairs still listed are tested
      const bool last = i0 >= n || __shfl_sync(0xffffffffu, *ncomp, 0) == 1;
      const uint32_t i = i0 + (tid & 31);
      const bool act = i < n && !last;
      int sx = 0, sy = 0, sz = 0;
      uint32_t ri = 0;
      if (act) {
        const uint64_t pg = A.run_g[f + i];
        const int gx = (int)(pg & kM21), gy = (int)((pg >> 21) & kM21), gz = (int)(pg >> 42);
        sx = gx - div_k(gx, g) * k;
        sy = gy - div_k(gy, g) * k;
        sz = gz - div_k(gz, g) * k;
        ri = lfind(lpar, i);  // may go stale: re-found before a pair is listed
      }
      const bool main = pass >= 1 && act && ri == lfind(lpar, *vmain);
      // columns within reach, the near ones (|dx| <= 1) and a's own
      const uint32_t reach = bit_span(max(sx - W, 0), min(sx + W, k - 1));
      const uint32_t near = bit_span(max(sx - 1, 0), min(sx + 1, k - 1));
      const uint32_t own = 1u << sx, after = sx == 31 ? 0u : (0xffffffffu << (sx + 1));
      // the forward rows (dz, dy) in order, from (0, 0) to (Wp, Wp)
      for (int dz = 0, dy = 0; dz <= (last ? 0 : Wp); dy == Wp ? (dz++, dy = -Wp) : dy++) {
        const int ty = sy + dy, tz = sz + dz, off = abs(dy) + dz;  // off 0: a's own row
        if (pass == 0 && off > 1 && !last) continue;
        uint32_t occ = 0, bits = 0, before = 0;
        if (act && ty >= 0 && ty < k && tz < k) {
          uint32_t m = max(abs(dy), dz) > 1 ? reach : pass == 2 ? reach & ~near : near;
          if (pass == 0 && off == 1) m = own;
          if (pass == 1 && off <= 1) m &= off == 0 ? 0u : ~own;
          if (off == 0) m &= after;  // forward only
          const uint32_t row = (uint32_t)(tz * k + ty);
          occ = rows[row];
          bits = (main ? rest[row] : occ) & m;
          before = pref[row];
        }
        while (last || __any_sync(0xffffffffu, bits)) {
          bool apart = false;
          uint32_t lj = 0;
          if (bits) {
            lj = before + __popc(occ & ((bits & -bits) - 1u));
            bits &= bits - 1u;
            st.cand++;
            const uint32_t rj = lfind(lpar, lj);
            if (rj != ri) ri = lfind(lpar, i);
            apart = rj != ri;
            if (!apart) st.skips++;
          }
          push_pairs<PT, FP32, VL>(A, uf, pairs, npair, apart, f + i, f + lj, last, st);
          if (last) break;
        }
        if (last) break;
      }
      if (last) break;
    }
    sync();
  }
  // joined to its local root through the global union-find: the sparse
  // kernel runs at the same time and may have hooked a cell of this top cell
  for (uint32_t i = tid; i < n; i += nt) {
    const uint32_t r = f + lfind(lpar, i);
    if (r != f + i && atomicCAS(parent + f + i, f + i, r) != f + i)
      uf_union(parent, f + i, r, A.ctr, g.union_cap);
  }
  // the rows stay for the queued cells' path, which looks up this top cell's
  // fine cells from its neighbours: a word per plane (bit y: row y holds fine
  // cells) and one of those outside the main component, a fine cell of the
  // main component, then per row its occupancy, the index of its first fine
  // cell and its occupancy outside the main component
  find_main();
  uint4 *gr = grows + (uint64_t)slot * rows_stride;
  uint32_t *head = reinterpret_cast<uint32_t *>(gr);
  for (uint32_t z = tid; z < (uint32_t)k; z += nt) {
    uint32_t plane = 0, prest = 0;
    for (int y = 0; y < k; y++) {
      plane |= (rows[z * k + y] != 0u ? 1u : 0u) << y;
      prest |= (rest[z * k + y] != 0u ? 1u : 0u) << y;
    }
    head[z] = plane;
    head[k + z] = prest;
  }
  if (tid == 0) head[2 * k] = f + *vmain;
  for (uint32_t j = tid; j < nrow; j += nt)
    gr[row_head(k) + j] = make_uint4(rows[j], f + pref[j], rest[j], 0u);
  sync();
}

// The dense top cells.  The big ones (more than big_min fine cells, listed
// in `big`) go first, one per CTA, so that the largest, which bound the
// kernel's length, start early and have many threads; then each warp takes
// the small ones one at a time, with its own slice of `lstride` words of
// shared memory (parents and bit rows).  Both kinds are taken from atomic counters: their sizes
// differ widely.
template <class PT, bool FP32, bool VL>
__global__ void __launch_bounds__(128) k_befriend_dense(
    const PairArgs<PT, FP32> A, uint64_t k3all, const uint2 *__restrict__ dense_range,
    const uint32_t *__restrict__ big, DevScal *sc, uint32_t nd_cap, uint4 *__restrict__ grows,
    uint32_t kk, uint32_t rows_stride, uint32_t *parent, uint32_t lstride, uint32_t big_min) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  extern __shared__ uint32_t smem[];
  __shared__ uint32_t s_slot;
  __shared__ uint2 s_pairs[4][kPairSlots];
  uint2 *pairs = s_pairs[threadIdx.x >> 5];
  const uint32_t nd = min(sc->nd, nd_cap), nbig = sc->nbig;
  const uint32_t lane = threadIdx.x & 31;
  uint32_t *own = smem + (size_t)(threadIdx.x >> 5) * lstride;
  BfStats st;
  bool cta = true;
  while (true) {
    uint32_t slot = 0;
    if (cta) {
      if (threadIdx.x == 0) {
        const uint32_t b = atomicAdd(&sc->next_big, 1u);
        s_slot = b < nbig ? big[b] : kNone;
      }
      __syncthreads();
      slot = s_slot;
      __syncthreads();
      if (slot == kNone) {
        cta = false;
        continue;
      }
    } else {
      if (lane == 0) slot = atomicAdd(&sc->next_dense, 1u);
      slot = __shfl_sync(0xffffffffu, slot, 0);
      if (slot >= nd) break;
      const uint2 fr = dense_range[slot];
      if (fr.y - fr.x > big_min) continue;
    }
    dense_top<PT, FP32, VL>(A, slot, cta ? smem : own, cta, pairs, k3all, dense_range, grows, kk,
                            rows_stride, parent, st);
    st.spill(A.ctr);
  }
  st.flush(A.ctr);
}

// The forward top cells (and a's own, bit 0) that hold cells within W of fine
// cell a: along an axis the lower (upper) neighbour when a lies within W cells
// of that face and the neighbour exists.
__device__ __forceinline__ uint32_t reached_tops(const Geom &g, int W, const int (&t)[3],
                                                 const int (&s)[3]) {
  // the neighbours (bits in kFwd's order) at offset -1, 0 and +1 along each axis
  constexpr uint32_t at[3][3] = {
      {0x0924, 0x1249, 0x2492},
      {0x00e0, 0x0703, 0x381c},
      {0x0000, 0x001f, 0x3fe0}};
  uint32_t m = 0x3fffu;
#pragma unroll
  for (int a = 0; a < 3; a++)
    m &= at[a][1] | (s[a] < W && t[a] > 0 ? at[a][0] : 0u) |
         (s[a] >= g.k - W && t[a] + 1 < g.T[a] ? at[a][2] : 0u);
  return m;
}

// A warp's candidate (a, b) pairs: fewer than 32 are left over when 32 more may
// be added.
constexpr uint32_t kListSlots = 64;

// Candidates of fine cell a are the fine cells b > a (key order, so each
// unordered pair is visited once) within W fine cells on every axis; they
// live in a's top cell (after a) and the 13 forward top cells.
//
// The sparse path: pairs of a fine cell and a top cell in its reach ("items",
// about two per cell).  A warp takes 32 fine cells, one per lane, and lists
// their items; it takes the listed items 32 at a time, one per lane: an item
// of a dense top cell is queued for k_befriend_cross (a's own top cell, when
// dense, is k_befriend_dense's), the fine cells of a sparse one that lie in
// reach are listed as candidates; those are compared with a's root 32 at a
// time, and the pairs in different components are tested 32 at a time
// (drain_pairs).  Every level thus works with full warps and keeps 32 or more
// reads in flight, where a thread per fine cell would step through 14
// neighbours of which two are in reach.  Bound by read latency (long-scoreboard
// stalls; 40 registers and 6 CTAs per SM, with the pair tests in a call, were no
// faster).  At half the 256^3 box (ncu, cold): a thread per fine cell here with
// whole cells queued for the two phases below, their sparse neighbours read in
// each, took 0.32 + 0.18 + 0.21 ms; this split 0.33 + 0.07 + 0.06 ms.

template <class PT, bool FP32, bool VL>
__global__ void __launch_bounds__(kT, 4) k_befriend_sparse(
    const PairArgs<PT, FP32> A, DevScal *sc, const uint2 *__restrict__ top_range,
    const uint32_t *__restrict__ top_slot, uint32_t *parent, uint32_t *__restrict__ q_cell,
    uint32_t *__restrict__ q_top, uint32_t q_cap, uint32_t dense_min) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const uint32_t R = sc->R;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5, below = (1u << lane) - 1u;
  // {fine cell, forward neighbour (below 14) or 15 + distance in key order of a
  // fine cell in its own top cell}
  __shared__ uint2 s_item[kT / 32][kListSlots];
  __shared__ uint2 s_cand[kT / 32][kListSlots];  // {fine cell, candidate}
  __shared__ uint2 s_pairs[kT / 32][kPairSlots];
  uint2 *items = s_item[wid], *cands = s_cand[wid], *pairs = s_pairs[wid];
  const GlobalUF uf{parent};
  uint32_t nitem = 0, ncand = 0, npair = 0;
  BfStats st;
  // Warps take 32 to 128 consecutive fine cells at a time from a counter: the
  // work per cell varies a lot across the box (clumps, empty neighbourhoods).
  // Whole CTAs taking 1024 cells, with two barriers a chunk, were 15 % slower.
  const uint32_t warps = gridDim.x * (kT / 32);
  const uint32_t step = R >= warps * 256 ? 128u : 32u;
  while (true) {
    st.spill(A.ctr);
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&sc->next_simple, step);
    base = __shfl_sync(0xffffffffu, base, 0);
    // past the last chunk, what is left in the lists
    const bool last = base >= R;
    const uint32_t end = last ? base + 1 : min(base + step, R);
    for (uint32_t a0 = base; a0 < end || last; a0 += 32) {
      uint32_t tops = 0, own = 0;  // own: bit d, fine cell a + 1 + d of a's top cell
      {
        const bool act = !last && a0 + lane < end;
        uint64_t pg = 0, t_own = ~0ull;
        int W = 0;
        if (act) {
          const BoxDev &bx = A.boxes[A.run_box[a0 + lane]];
          const Geom &g = bx.g;
          pg = A.run_g[a0 + lane];
          const int c[3] = {(int)(pg & kM21), (int)((pg >> 21) & kM21), (int)(pg >> 42)};
          const int t[3] = {div_k(c[0], g), div_k(c[1], g), div_k(c[2], g)};
          const int f[3] = {c[0] - t[0] * g.k, c[1] - t[1] * g.k, c[2] - t[2] * g.k};
          W = g.W;
          tops = reached_tops(g, W, t, f);
          t_own = bx.top_base + ((uint64_t)t[2] * g.T[1] + t[1]) * g.T[0] + t[0];
        }
        // The rest of a's top cell lies in the following lanes, unless it goes on
        // past the warp's last cell (then it is an item like the others).
        // A top cell that starts here and has at most dense_min fine cells is
        // sparse; of the others the slot tells.
        const uint64_t t_prev = __shfl_up_sync(0xffffffffu, t_own, 1);
        const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0 || t_own != t_prev);
        const uint32_t acts = __ballot_sync(0xffffffffu, act);
        const uint32_t after = heads & ~((2u << lane) - 1u);  // (none past the last lane)
        const bool whole = act && after && (acts >> (__ffs(after) - 1) & 1u);
        uint32_t n = 0;
        if (whole) {
          tops &= ~1u;
          n = (uint32_t)__ffs(after) - 2u - lane;
          if (n) {
            const uint32_t first = 31u - (uint32_t)__clz((int)(heads & ((2u << lane) - 1u)));
            if ((first == 0 || lane - first + n + 1 > dense_min) && top_slot[t_own] != kNone) n = 0;
          }
        }
        const uint32_t most = __reduce_max_sync(0xffffffffu, n);
        for (uint32_t d = 1; d <= most; d++) {
          const uint64_t qg = __shfl_down_sync(0xffffffffu, pg, d);
          if (d <= n &&
              max(abs((int)(qg & kM21) - (int)(pg & kM21)),
                  max(abs((int)((qg >> 21) & kM21) - (int)((pg >> 21) & kM21)),
                      abs((int)(qg >> 42) - (int)(pg >> 42)))) <= W)
            own |= 1u << (d - 1);
        }
      }
      do {
        {
          const uint32_t m = __ballot_sync(0xffffffffu, (tops | own) != 0);
          if (own) {
            items[nitem + __popc(m & below)] = make_uint2(a0 + lane, 15u + (uint32_t)__ffs(own));
            own &= own - 1u;
          } else if (tops) {
            items[nitem + __popc(m & below)] = make_uint2(a0 + lane, (uint32_t)__ffs(tops) - 1u);
            tops &= tops - 1u;
          }
          nitem += __popc(m);
        }
        if (nitem < 32 && !last) continue;
        // the last 32 items, one per lane
        __syncwarp();
        const uint32_t n = min(nitem, 32u);
        nitem -= n;
        uint32_t a = 0, r0 = 0, cnt = 0, slot = kNone, nb = 0;
        int gx = 0, gy = 0, gz = 0, W = 0;
        if (lane < n) {
          const uint2 it = items[nitem + lane];
          a = it.x;
          nb = it.y;
          const BoxDev &bx = A.boxes[A.run_box[a]];
          const Geom &g = bx.g;
          const uint64_t pg = A.run_g[a];
          gx = (int)(pg & kM21);
          gy = (int)((pg >> 21) & kM21);
          gz = (int)(pg >> 42);
          W = g.W;
          if (nb < 14) {
            const uint64_t tb = bx.top_base +
                                ((uint64_t)(div_k(gz, g) + kFwd[nb][2]) * g.T[1] +
                                 (uint64_t)(div_k(gy, g) + kFwd[nb][1])) * g.T[0] +
                                (uint64_t)(div_k(gx, g) + kFwd[nb][0]);
            const uint2 tr = top_range[tb];
            slot = top_slot[tb];
            r0 = nb == 0 ? a + 1 : tr.x;
            cnt = tr.y > r0 ? tr.y - r0 : 0u;
            if (nb == 0 && slot != kNone) cnt = 0;  // k_befriend_dense's
          } else {
            r0 = a + nb - 15u;  // a fine cell of a's own top cell, in reach
            cnt = 1;
          }
        }
        __syncwarp();  // (read before other lanes list items there again)
        const bool dense = cnt != 0 && slot != kNone;
        const uint32_t qm = __ballot_sync(0xffffffffu, dense);
        if (qm) {
          unsigned long long at = 0;  // (may pass 2^32: no early place is taken twice)
          if (lane == 0) at = atomicAdd(&sc->qcount, (unsigned long long)__popc(qm));
          at = __shfl_sync(0xffffffffu, at, 0) + __popc(qm & below);
          if (dense && at < q_cap) {  // (past the queue's end the cells are read one by one)
            q_cell[at] = a;
            q_top[at] = nb << 28 | slot;
            cnt = 0;
          }
        }
        for (uint32_t i0 = 0; __any_sync(0xffffffffu, i0 < cnt) || (last && i0 == 0); i0 += 32) {
          uint32_t todo = 0;  // bit i: fine cell r0 + i0 + i is within reach
          if (i0 < cnt) {
            const uint32_t m = min(cnt - i0, 32u);
#pragma unroll 4
            for (uint32_t u = 0; u < m; u++) {
              const uint64_t qg = A.run_g[r0 + i0 + u];
              const int cheb =
                  max(abs((int)(qg & kM21) - gx),
                      max(abs((int)((qg >> 21) & kM21) - gy), abs((int)(qg >> 42) - gz)));
              if (cheb <= W) todo |= 1u << u;
            }
            st.scan += m;
          }
          const bool end_items = !__any_sync(0xffffffffu, i0 + 32 < cnt);
          do {
            const uint32_t m = __ballot_sync(0xffffffffu, todo != 0);
            if (todo) {
              cands[ncand + __popc(m & below)] =
                  make_uint2(a, r0 + i0 + (uint32_t)__ffs(todo) - 1u);
              todo &= todo - 1u;
            }
            ncand += __popc(m);
            const bool flush = last && end_items && !__any_sync(0xffffffffu, todo != 0);
            if (ncand < 32 && !flush) continue;
            do {
              // the last 32 candidates against their cells' roots
              __syncwarp();
              const uint32_t nc = min(ncand, 32u);
              ncand -= nc;
              bool apart = false;
              uint2 c = make_uint2(0u, 0u);
              if (lane < nc) {
                c = cands[ncand + lane];
                st.cand++;
                st.steps += 2;
                uint32_t ra = __ldcg(parent + c.x), rb = __ldcg(parent + c.y);
                if (rb != ra && rb != c.y) rb = uf_find_n(parent, rb, st.steps);
                if (rb != ra && ra != c.x) ra = uf_find_n(parent, ra, st.steps);
                apart = rb != ra;
                if (!apart) st.skips++;
              }
              __syncwarp();  // (read before other lanes list candidates there again)
              push_pairs<PT, FP32, VL>(A, uf, pairs, npair, apart, c.x, c.y, flush && ncand == 0,
                                       st);
            } while (flush && ncand);
          } while (__any_sync(0xffffffffu, todo != 0));
        }
      } while (__any_sync(0xffffffffu, (tops | own) != 0));
      if (last) break;
    }
    if (last) break;
  }
  st.flush(A.ctr);
}

// The queued items: fine cells and the dense forward top cells in their reach.
// PHASE 0 visits the candidates within one fine cell, PHASE 1 the farther
// ones, so that a dense neighbourhood is joined (and compressed) before its far
// pairs are tried and most of those are found joined.
//
// The kernel is bound by the latency of its table reads and by instruction
// issue, so a warp works its items off in three levels, each with all lanes
// busy and many reads in flight.  It takes 32 items, one per lane (or 32 / G
// items of G lanes each when the queue is short, so that it still fills the
// chip; one atomic per grab).  1: the neighbour's plane words (bit y: row y of
// the plane holds fine cells) give the window's non-empty rows -- of those
// outside the neighbour's main component when that is joined to the cell
// already, as it mostly is inside clumps -- one bit each, listed.  2: the listed
// rows are taken 32 at a time, one per lane: the row's word gives the
// candidates, each compared with its cell's root.  3: candidates in another
// component are tested 32 at a time (drain_pairs).  Most rows are empty, hence
// the plane words, and most candidates inside clumps are joined already, hence
// the main components: without them a far phase over whole cells issued 1.4
// times the instructions.  Befriending of the 256^3 box: 2.80 ms with a warp per
// cell and a lane per window slot, 1.76 ms with 32 cells a warp, 1.20 ms with
// items of dense neighbours only; of the 512^3 box at the 1024^3 box's
// parameters 36.5, 21.5 and 13.6 ms.
constexpr int kPlanes = 5;  // plane words read at a time
// floor(i / d) = i * kDiv[d] >> 16 for i < 1200, d <= 32
__constant__ uint32_t kDiv[33] = {
    0,    65536, 32769, 21846, 16385, 13108, 10923, 9363, 8193, 7282, 6554,
    5958, 5462,  5042,  4682,  4370,  4097,  3856,  3641, 3450, 3277, 3121,
    2979, 2850,  2731,  2622,  2521,  2428,  2341,  2260, 2185, 2115, 2049};

template <class PT, bool FP32, bool VL, int PHASE>
__global__ void __launch_bounds__(kT, 3) k_befriend_cross(
    const PairArgs<PT, FP32> A, const uint32_t *__restrict__ q_cell,
    const uint32_t *__restrict__ q_top, uint32_t q_cap, DevScal *sc,
    const uint4 *__restrict__ grows, uint32_t rows_stride, uint32_t *parent) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  __shared__ uint2 s_pairs[kT / 32][kPairSlots];
  // listed rows: {index of the row's word (+ 2^31: only the cells outside the
  // main component), columns within reach, fine cell, its root}
  __shared__ uint4 s_row[kT / 32][kListSlots];
  uint2 *pairs = s_pairs[threadIdx.x >> 5];
  uint4 *rows = s_row[threadIdx.x >> 5];
  const GlobalUF uf{parent};
  const uint32_t NQ = (uint32_t)min(sc->qcount, (unsigned long long)q_cap);
  if (NQ == 0) return;
  uint32_t *next = PHASE == 0 ? &sc->next0 : &sc->next1;
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
  // lanes per item: the fewest (1, 2, 4, 8) that give every thread of the grid work
  int lg = 0;
  while (lg < 3 && ((uint64_t)NQ << lg) < (uint64_t)gridDim.x * blockDim.x) lg++;
  const uint32_t G = 1u << lg;
  // a lane's share of its item's rows: every G-th
  const uint64_t share = (lg == 0 ? ~0ull : lg == 1 ? 0x5555555555555555ull
                          : lg == 2 ? 0x1111111111111111ull : 0x0101010101010101ull)
                         << (lane & (G - 1));
  uint32_t npair = 0, nrow = 0;
  BfStats st;
  while (true) {
    st.spill(A.ctr);
    uint32_t q0 = 0;
    if (lane == 0) q0 = atomicAdd(next, 32u >> lg);
    q0 = __shfl_sync(0xffffffffu, q0, 0);
    const bool last = q0 >= NQ;  // past the last items, what is left in the lists
    const uint32_t qi = q0 + (lane >> lg);
    const uint4 *gr = nullptr;
    bool rest = false;                   // only cells outside its main component
    uint32_t a = 0, ra = 0, cnt = 0, chunk = 32, reach = 0, inner = 0;
    int k = 1, cx = 0, cy = 0, cz = 0;   // a in the neighbour's own fine coordinates
    int y0 = 0, ny = 1, z0 = 0;          // the window's rows there
    if (qi < NQ && !last) {
      a = q_cell[qi];
      const uint32_t it = q_top[qi], nb = it >> 28;
      gr = grows + (uint64_t)(it & 0x0fffffffu) * rows_stride;
      const Geom &g = A.boxes[A.run_box[a]].g;
      k = g.k;
      const int W = PHASE == 0 ? 1 : g.W;
      const uint64_t pg = A.run_g[a];
      const int gx = (int)(pg & kM21), gy = (int)((pg >> 21) & kM21), gz = (int)(pg >> 42);
      cx = gx - (div_k(gx, g) + kFwd[nb][0]) * k;
      cy = gy - (div_k(gy, g) + kFwd[nb][1]) * k;
      cz = gz - (div_k(gz, g) + kFwd[nb][2]) * k;
      const int x0 = max(cx - W, 0), x1 = min(cx + W, k - 1);
      y0 = max(cy - W, 0);
      ny = min(cy + W, k - 1) - y0 + 1;
      z0 = max(cz - W, 0);
      const int nz = min(cz + W, k - 1) - z0 + 1;
      if (x0 <= x1 && ny > 0 && nz > 0) {  // (PHASE 0 may not reach the neighbour)
        reach = bit_span(x0, x1);
        // the near columns, which were PHASE 0's in the rows within one row of a
        if (PHASE == 1 && cx >= -1 && cx <= k)
          inner = bit_span(max(cx - 1, 0), min(cx + 1, k - 1));
        // cells of the neighbour's main component are joined to a already?
        ra = __ldcg(parent + a);
        uint32_t rm = __ldcg(parent + reinterpret_cast<const uint32_t *>(gr)[2 * k]);
        st.steps += 2;
        if (rm != ra) {
          rm = uf_find_n(parent, rm, st.steps);
          if (rm != ra) ra = uf_find_n(parent, ra, st.steps);
        }
        rest = rm == ra;
        cnt = (uint32_t)(ny * nz);
        // whole planes, as many as kPlanes and 64 bits take
        chunk = (uint32_t)ny * min((64u * kDiv[ny]) >> 16, (uint32_t)kPlanes);
      }
    }
    for (uint32_t i0 = 0; __any_sync(0xffffffffu, i0 < cnt) || (last && i0 == 0); i0 += chunk) {
      uint64_t todo = 0;  // bit i: row i0 + i of the window is to be listed
      if (i0 < cnt) {
        const int zz = (int)((i0 * kDiv[ny]) >> 16);
        const uint32_t *planes =
            reinterpret_cast<const uint32_t *>(gr) + (rest ? k : 0) + z0 + zz;
        const uint32_t span = bit_span(0, ny - 1), m = min(chunk, cnt - i0);
#pragma unroll
        for (int u = 0; u < kPlanes; u++)
          if (u * ny < (int)m) todo |= (uint64_t)((planes[u] >> y0) & span) << (u * ny);
        todo &= share;
        st.window += __popcll(todo);
      }
      const bool end_items = !__any_sync(0xffffffffu, i0 < cnt && i0 + chunk < cnt);
      do {
        bool add = todo != 0;
        uint4 e = make_uint4(0u, 0u, a, ra);
        if (add) {
          const uint32_t i = i0 + (uint32_t)__ffsll((long long)todo) - 1u;
          todo &= todo - 1u;
          const int zz = (int)((i * kDiv[ny]) >> 16), z = z0 + zz, y = y0 + (int)i - zz * ny;
          e.x = (uint32_t)(gr - grows) + (uint32_t)(row_head(k) + z * k + y) +
                (rest ? 0x80000000u : 0u);
          e.y = PHASE == 1 && max(abs(y - cy), abs(z - cz)) <= 1 ? reach & ~inner : reach;
          add = e.y != 0;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, add);
        if (add) rows[nrow + __popc(m & below)] = e;
        nrow += __popc(m);
        const bool flush = last && end_items && !__any_sync(0xffffffffu, todo != 0);
        if (nrow < 32 && !flush) continue;
        // the last 32 listed rows, one per lane
        __syncwarp();
        const uint32_t n = min(nrow, 32u);
        nrow -= n;
        uint32_t bits = 0, occ = 0, first = 0, ca = 0, cr = 0;
        if (lane < n) {
          const uint4 w = rows[nrow + lane];
          const uint4 word = grows[w.x & 0x7fffffffu];
          occ = word.x;
          bits = (w.x >> 31 ? word.z : occ) & w.y;
          first = word.y;
          ca = w.z;
          cr = w.w;
        }
        do {
          bool apart = false;
          uint32_t b = 0;
          if (bits) {
            b = first + __popc(occ & ((bits & -bits) - 1u));
            bits &= bits - 1u;
            st.cand++;
            st.steps++;
            // (PHASE 1: the cached parent may be an older one, which is still
            // in the candidate's component)
            uint32_t rb = PHASE == 1 ? __ldca(parent + b) : __ldcg(parent + b);
            if (rb != cr && rb != b) rb = uf_find_n(parent, rb, st.steps);
            // cr may have been hooked since; it stays in its cell's component
            if (rb != cr) cr = uf_find_n(parent, cr, st.steps);
            apart = rb != cr;
            if (!apart) st.skips++;
          }
          const bool more = __any_sync(0xffffffffu, bits != 0);
          push_pairs<PT, FP32, VL>(A, uf, pairs, npair, apart, ca, b, flush && !more, st);
        } while (__any_sync(0xffffffffu, bits != 0));
        __syncwarp();
      } while (__any_sync(0xffffffffu, todo != 0));
    }
    if (last) break;
  }
  st.flush(A.ctr);
}

__global__ void __launch_bounds__(kT) k_compress(uint32_t *parent,
                                                 const DevScal *__restrict__ sc) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const uint32_t R = sc->R;
  for (int64_t r = gtid(); r < R; r += gstride()) parent[r] = uf_find(parent, (uint32_t)r);
}

// ---------------------------------------------------------------------------
// Segmented reductions over cell-ordered particles.
// ---------------------------------------------------------------------------

// Lanes of a warp holding the same key in adjacent lanes form a segment; the
// segment's first lane receives the segment's sum of v (and min of m).
template <int NV>
__device__ __forceinline__ bool warp_segments(uint32_t key, double (&v)[NV], uint32_t &m) {
  const int lane = threadIdx.x & 31;
  const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
  const bool head = lane == 0 || prev != key;
  const uint32_t heads = __ballot_sync(0xffffffffu, head);
  const uint32_t seg = __popc(heads & ((2u << lane) - 1u));  // 1-based segment id
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t oseg = __shfl_down_sync(0xffffffffu, seg, d);
    const bool take = (lane + d < 32) && oseg == seg;
#pragma unroll
    for (int c = 0; c < NV; c++) {
      const double t = __shfl_down_sync(0xffffffffu, v[c], d);
      if (take) v[c] += t;
    }
    const uint32_t om = __shfl_down_sync(0xffffffffu, m, d);
    if (take) m = min(m, om);
  }
  return head;
}

__device__ __forceinline__ bool warp_segments_count(uint32_t key, uint32_t &cnt) {
  const int lane = threadIdx.x & 31;
  const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
  const bool head = lane == 0 || prev != key;
  const uint32_t heads = __ballot_sync(0xffffffffu, head);
  const uint32_t seg = __popc(heads & ((2u << lane) - 1u));
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t oseg = __shfl_down_sync(0xffffffffu, seg, d);
    const uint32_t oc = __shfl_down_sync(0xffffffffu, cnt, d);
    if ((lane + d < 32) && oseg == seg) cnt += oc;
  }
  return head;
}

// After the last union: each cell's root as its parent, and the roots' group
// sizes, a cell's run of particles at a time: half the elements of a count by
// particle and none of its look-ups.  The walk to the root only reads, so that a
// cell's parent is written by its own thread alone: the kernels that follow take
// it as the root without a find, and a halving find's late store of an ancestor
// over the root would take the cell out of its group's sums and membership.
// The groups' heads are found for the
// candidates alone, by k_group_sums, not with an atomic per group here.  Bound
// by the parents' reads and the counts' atomics.  Befriending, groups and sums
// with a compression, then counts and heads by particle, and so: 256^3 box
// 1.52 and 1.46 ms, 512^3 box 16.06 and 15.73, 50M lightcone 4.52 and 4.41.
__global__ void __launch_bounds__(kT) k_compress_count(uint32_t *parent,
                                                       const uint32_t *__restrict__ run_start,
                                                       const DevScal *__restrict__ sc,
                                                       uint32_t *__restrict__ count) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const int64_t R = sc->R;
  const int64_t n_iter = (R + 31) / 32 * 32;
  for (int64_t r = gtid(); r < n_iter; r += gstride()) {
    const bool valid = r < R;
    uint32_t root = kNone, c = 0;
    if (valid) {
      root = uf_root(parent, (uint32_t)r);
      parent[r] = root;
      c = run_start[r + 1] - run_start[r];
    }
    const bool h = warp_segments_count(root, c);
    if (valid && h) atomicAdd(count + root, c);
  }
}

// Subsampling (FOF.c:205-284): every original particle inside its box's
// domain ([lo, hi) per axis, [lo, hi] on the axes of `closed`) is kept when its uniform is
// below its group's rate -- samp_in for groups of at least Nphalomin
// processed particles (FOF.c:202), samp_out for the others.  The uniform is
// the top 53 bits of SplitMix64's output mix (Steele, Lea & Flood 2014) of
// key ^ (seed * 0xD1B54A32D192ED03), key = the particle's ID or its input
// index, so a particle's draw depends on nothing but the seed and itself.
__device__ __forceinline__ double sample_uniform(uint64_t seed, uint64_t key) {
  uint64_t z = key ^ (seed * 0xD1B54A32D192ED03ull);
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * 0x1.0p-53;
}

template <class PT>
__global__ void __launch_bounds__(kT) k_subsample(
    const uint32_t *__restrict__ run_of, const uint32_t *__restrict__ parent,
    const uint32_t *__restrict__ count, const uint32_t *__restrict__ perm,
    const SPos<PT> *__restrict__ spos, const uint16_t *__restrict__ run_box,
    const BoxDev *__restrict__ boxes, const uint32_t *__restrict__ boxd, int nbox,
    const DevScal *__restrict__ sc, const uint64_t *__restrict__ ids, double samp_in,
    double samp_out, uint64_t seed, int closed, uint8_t *__restrict__ samp) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const int64_t np = sc->np;
  for (int64_t i = gtid(); i < np; i += gstride()) {
    const uint32_t run = run_of[i];
    const int b = run_box[run];
    if (perm[i] - boxd[4 * nbox + b] >= boxd[2 * nbox + b]) continue;  // an image
    const Geom &g = boxes[b].g;
    const SPos<PT> sp = spos[i];
    const double x[3] = {as_d(sp.x), as_d(sp.y), as_d(sp.z)};
    bool inside = true;
#pragma unroll
    for (int a = 0; a < 3; a++)
      inside &= x[a] >= g.lo[a] && (((closed >> a) & 1) ? x[a] <= g.hi[a] : x[a] < g.hi[a]);
    if (!inside) continue;
    const bool in = !((double)count[parent[run]] < g.nphalomin);
    const double rate = in ? samp_in : samp_out;
    if (!(rate > 0.0)) continue;
    const uint64_t key = ids ? ids[sp.src] : (uint64_t)sp.src;
    if (sample_uniform(seed, key) < rate) samp[sp.src] = in ? 1 : 2;
  }
}

// Candidate halos: roots of at least Nphalomin members (FOF.c:202), each
// given an index from a counter (the catalog is put in head order later, so
// the candidates' order does not matter); counts the roots (groups).
__global__ void __launch_bounds__(kT) k_cand_pick(const uint32_t *__restrict__ parent,
                                                  const uint32_t *__restrict__ count,
                                                  const uint16_t *__restrict__ run_box,
                                                  const BoxDev *__restrict__ boxes,
                                                  DevScal *sc,
                                                  uint32_t *__restrict__ cand_of_root,
                                                  uint32_t *__restrict__ cand_root,
                                                  unsigned long long *ngroups) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const uint32_t R = sc->R;
  const int lane = threadIdx.x & 31;
  unsigned long long roots = 0;
  for (int64_t r0 = gtid() - lane; r0 < (int64_t)R; r0 += gstride()) {
    const int64_t r = r0 + lane;
    bool cand = false;
    if (r < (int64_t)R) {
      const bool root = parent[r] == (uint32_t)r;
      roots += root;
      cand = root && !((double)count[r] < boxes[run_box[r]].g.nphalomin);
    }
    const uint32_t ci = warp_slot(cand, &sc->nc);
    if (cand) {
      cand_of_root[r] = ci;
      cand_root[ci] = (uint32_t)r;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) roots += __shfl_down_sync(0xffffffffu, roots, d);
  if (lane == 0 && roots) atomicAdd(ngroups, roots);
}

// Property sums per candidate halo, in double as Output_Halos does
// (FOF.c:806-832): 6 first moments, then 6 position and 6 velocity second
// moments when INERTIA / DISPERSION are asked for; and its head, the lowest
// processing index of its particles.
template <class PT, int NS>
__global__ void __launch_bounds__(kT) k_group_sums(
    const uint32_t *__restrict__ run_of, const uint32_t *__restrict__ parent,
    const uint32_t *__restrict__ cand_of_root, const uint16_t *__restrict__ run_box,
    const BoxDev *__restrict__ boxes, const SPos<PT> *__restrict__ spos,
    const uint32_t *__restrict__ perm, const DevScal *__restrict__ sc, int props,
    double *__restrict__ sums, uint32_t *__restrict__ head, uint32_t *__restrict__ warn) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const int64_t np = sc->np;
  const int64_t n_iter = (np + 31) / 32 * 32;
  for (int64_t i = gtid(); i < n_iter; i += gstride()) {
    uint32_t ci = kNone, m = kNone;
    double v[NS];
#pragma unroll
    for (int c = 0; c < NS; c++) v[c] = 0.0;
    if (i < np) {
      const uint32_t run = run_of[i];
      ci = cand_of_root[parent[run]];
      if (ci != kNone) {
        const BoxDev &bx = boxes[run_box[run]];
        const Geom &g = bx.g;
        const SPos<PT> p = spos[i];
        m = perm[i];
        const double x = (double)p.x, y = (double)p.y, z = (double)p.z;
        const uint64_t li = 3 * ((uint64_t)p.src - bx.in_base);
        double vx, vy, vz;
        if (bx.vel_f64) {
          const double *vel = static_cast<const double *>(bx.vel);
          vx = vel[li]; vy = vel[li + 1]; vz = vel[li + 2];
        } else {
          const float *vel = static_cast<const float *>(bx.vel);
          vx = (double)vel[li]; vy = (double)vel[li + 1]; vz = (double)vel[li + 2];
        }
        v[0] = x; v[1] = y; v[2] = z; v[3] = vx; v[4] = vy; v[5] = vz;
        if constexpr (NS >= 12) {
          if (props & 1) {
            v[6] = __dmul_rn(x, x); v[7] = __dmul_rn(y, y); v[8] = __dmul_rn(z, z);
            v[9] = __dmul_rn(x, y); v[10] = __dmul_rn(x, z); v[11] = __dmul_rn(y, z);
          }
        }
        if constexpr (NS >= 18) {
          v[12] = __dmul_rn(vx, vx); v[13] = __dmul_rn(vy, vy); v[14] = __dmul_rn(vz, vz);
          v[15] = __dmul_rn(vx, vy); v[16] = __dmul_rn(vx, vz); v[17] = __dmul_rn(vy, vz);
        } else if constexpr (NS >= 12) {
          if (!(props & 1)) {
            v[6] = __dmul_rn(vx, vx); v[7] = __dmul_rn(vy, vy); v[8] = __dmul_rn(vz, vz);
            v[9] = __dmul_rn(vx, vy); v[10] = __dmul_rn(vx, vz); v[11] = __dmul_rn(vy, vz);
          }
        }
        // edge warning of Checkhalo (FOF.c:406-422)
        if (x - g.rmin[0] < g.maxlink || g.rmax[0] - x < g.maxlink ||
            y - g.rmin[1] < g.maxlink || g.rmax[1] - y < g.maxlink ||
            z - g.rmin[2] < g.maxlink || g.rmax[2] - z < g.maxlink)
          atomicOr(warn + ci, 1u);
      }
    }
    // stretches of background hold no candidate at all (256^3 box: 0.29 -> 0.27 ms,
    // 64 boxes 0.87 -> 0.76; two or four particles per step, their gathers in flight
    // together, were 10 and 20 % slower: fewer warps)
    if (!__any_sync(0xffffffffu, ci != kNone)) continue;
    const bool h = warp_segments<NS>(ci, v, m);
    if (h && ci != kNone) {
      atomicMin(head + ci, m);
      double *s = sums + (uint64_t)ci * NS;
#pragma unroll
      for (int c = 0; c < NS; c++) atomicAdd(s + c, v[c]);
    }
  }
}

// The catalog lists the owned halos by head.  Heads are distinct processing
// indices, so a halo's place is the number of owned heads below its own: one
// bit per processing index, counts of kHeadGroup of them, their prefix.  Three
// short kernels whatever the number of halos, where a sort of the heads took
// four to seven and a quarter of a small run's launches (64^3 box: catalog 0.075
// -> 0.028 ms; 512^3 box, 142M bits: 0.17 -> 0.20 ms of 35).
constexpr uint32_t kHeadGroup = 1024;  // 32 words of 32 heads

// Ownership (Checkhalo, FOF.c:394-401): centre of mass by division, kept iff
// inside [lo, hi) on every axis.  An owned candidate is listed (from a counter)
// with its head, which is marked in `marks`, and counted for its box.  (Past the
// capacity heads are not marked: the run is then repeated with more room.)
template <int NS>
__global__ void __launch_bounds__(kT) k_own_pick(const double *__restrict__ sums,
                                                 const uint32_t *__restrict__ cand_root,
                                                 const uint32_t *__restrict__ count,
                                                 const uint32_t *__restrict__ head,
                                                 const uint16_t *__restrict__ run_box,
                                                 const BoxDev *__restrict__ boxes,
                                                 DevScal *sc, uint32_t *__restrict__ own_head,
                                                 uint32_t *__restrict__ own_cand,
                                                 uint32_t *__restrict__ marks, uint32_t np_cap,
                                                 uint32_t *__restrict__ boxd, int nbox) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const uint32_t nc = sc->nc;
  const int lane = threadIdx.x & 31;
  for (int64_t c0 = gtid() - lane; c0 < (int64_t)nc; c0 += gstride()) {
    const int64_t c = c0 + lane;
    bool ok = false;
    uint32_t hd = 0;
    int b = 0;
    if (c < (int64_t)nc) {
      const uint32_t root = cand_root[c];
      b = run_box[root];
      const Geom &g = boxes[b].g;
      const double n = (double)count[root];
      ok = true;
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const double com = __ddiv_rn(sums[(uint64_t)c * NS + a], n);
        ok &= (com >= g.lo[a]) && (com < g.hi[a]);
      }
      hd = head[c];
      ok &= hd < np_cap;
    }
    const uint32_t o = warp_slot(ok, &sc->nh);
    if (ok) {
      own_head[o] = hd;
      own_cand[o] = (uint32_t)c;
      atomicOr(marks + (hd >> 5), 1u << (hd & 31));
      atomicAdd(&boxd[5 * nbox + b], 1u);
    }
  }
}

// Marked heads per group, one warp each.
__global__ void __launch_bounds__(kT) k_head_groups(const uint32_t *__restrict__ marks,
                                                    uint32_t ngroup,
                                                    uint32_t *__restrict__ group,
                                                    const DevScal *__restrict__ sc) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  for (int64_t i = gtid(); i < (int64_t)ngroup * 32; i += gstride()) {
    const uint32_t n = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(marks[i]));
    if ((i & 31) == 0) group[i >> 5] = n;
  }
}

// One CTA: exclusive prefix of the groups, in place, and each box's first
// catalog index: processing indices number the boxes one after another.
__global__ void __launch_bounds__(kScanT) k_head_scan(uint32_t *group, uint32_t ngroup,
                                                      uint32_t *boxd, int nbox,
                                                      const DevScal *__restrict__ sc) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  __shared__ uint2 s_warp[kScanT / 32];
  constexpr uint32_t kItems = 8;
  uint32_t carry = 0;
  for (uint32_t g0 = 0; g0 < ngroup; g0 += kScanT * kItems) {
    uint32_t v[kItems], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < kItems; q++) {
      const uint32_t g = g0 + threadIdx.x * kItems + q;
      v[q] = g < ngroup ? group[g] : 0u;
      sum += v[q];
    }
    uint2 total;
    uint32_t run = block_exclusive2(make_uint2(sum, 0u), s_warp, &total).x + carry;
#pragma unroll
    for (uint32_t q = 0; q < kItems; q++) {
      const uint32_t g = g0 + threadIdx.x * kItems + q;
      if (g < ngroup) group[g] = run;
      run += v[q];
    }
    carry += total.x;
  }
  carry = 0;
  for (int b0 = 0; b0 < nbox; b0 += kScanT) {
    const int b = b0 + (int)threadIdx.x;
    const uint32_t v = b < nbox ? boxd[5 * nbox + b] : 0u;
    uint2 total;
    const uint32_t ex = block_exclusive2(make_uint2(v, 0u), s_warp, &total).x;
    if (b < nbox) boxd[6 * nbox + b] = carry + ex;
    carry += total.x;
  }
}

// Halo records (Output_Halos, FOF.c:836-872): means by the reciprocal of n,
// second-moment combinations as written there, all in double, then float.
// The head is reported as an index into the box's own processing order.
template <int NS>
__global__ void __launch_bounds__(kT) k_catalog(const uint32_t *__restrict__ own_head,
                                                const uint32_t *__restrict__ own_cand,
                                                const uint32_t *__restrict__ marks,
                                                const uint32_t *__restrict__ group,
                                                const DevScal *__restrict__ sc,
                                                const double *__restrict__ sums,
                                                const uint32_t *__restrict__ cand_root,
                                                const uint32_t *__restrict__ count,
                                                const uint32_t *__restrict__ warn,
                                                const uint16_t *__restrict__ run_box,
                                                const uint32_t *__restrict__ boxd, int nbox,
                                                int props, int hs, float *__restrict__ out_props,
                                                uint32_t *__restrict__ head_out,
                                                uint32_t *__restrict__ cat_of_cand,
                                                unsigned long long *n_warn) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const uint32_t nh = sc->nh;
  for (int64_t i = gtid(); i < nh; i += gstride()) {
    const uint32_t c = own_cand[i], hd = own_head[i], word = hd >> 5;
    uint32_t h = group[hd / kHeadGroup] + __popc(marks[word] & ((1u << (hd & 31)) - 1u));
    for (uint32_t q = word & ~31u; q < word; q++) h += __popc(marks[q]);
    const uint32_t root = cand_root[c];
    const uint32_t n = count[root];
    const int b = run_box[root];
    const double *s = sums + (uint64_t)c * NS;
    const double inv = __ddiv_rn(1.0, (double)n);
    float *rec = out_props + (uint64_t)h * hs;
    int o = 0;
    rec[o++] = (float)n;
    for (int q = 0; q < 6; q++) rec[o++] = __double2float_rn(__dmul_rn(s[q], inv));
    int m = 6;
    if (props & 1) {
      const double xx = s[m], yy = s[m + 1], zz = s[m + 2], xy = s[m + 3], xz = s[m + 4],
                   yz = s[m + 5];
      const double X = s[0], Y = s[1], Z = s[2];
      rec[o++] = __double2float_rn(__dsub_rn(__dadd_rn(yy, zz), __dmul_rn(inv, __dadd_rn(__dmul_rn(Y, Y), __dmul_rn(Z, Z)))));
      rec[o++] = __double2float_rn(__dsub_rn(__dadd_rn(xx, zz), __dmul_rn(inv, __dadd_rn(__dmul_rn(X, X), __dmul_rn(Z, Z)))));
      rec[o++] = __double2float_rn(__dsub_rn(__dadd_rn(xx, yy), __dmul_rn(inv, __dadd_rn(__dmul_rn(X, X), __dmul_rn(Y, Y)))));
      rec[o++] = __double2float_rn(__dsub_rn(__dmul_rn(__dmul_rn(inv, X), Y), xy));
      rec[o++] = __double2float_rn(__dsub_rn(__dmul_rn(__dmul_rn(inv, X), Z), xz));
      rec[o++] = __double2float_rn(__dsub_rn(__dmul_rn(__dmul_rn(inv, Y), Z), yz));
      m += 6;
    }
    if (props & 2) {
      const double VX = s[3], VY = s[4], VZ = s[5];
      const double A[6] = {s[m], s[m + 1], s[m + 2], s[m + 3], s[m + 4], s[m + 5]};
      const double P[6] = {__dmul_rn(VX, VX), __dmul_rn(VY, VY), __dmul_rn(VZ, VZ),
                           __dmul_rn(VX, VY), __dmul_rn(VX, VZ), __dmul_rn(VY, VZ)};
      for (int q = 0; q < 6; q++)
        rec[o++] = __double2float_rn(__dmul_rn(__dsub_rn(A[q], __dmul_rn(P[q], inv)), inv));
    }
    head_out[h] = hd - boxd[4 * nbox + b];
    cat_of_cand[c] = h;
    if (warn[c]) atomicAdd(n_warn, 1ull);
  }
}

// Membership per input particle: the owned halo holding it (or one of its
// images) -- the lowest catalog index when a halo wider than the ghost shell
// leaves two owned copies -- then, in a second pass, the processing index of
// that copy (in its box's numbering) and its stored coordinates.
template <class PT>
__global__ void __launch_bounds__(kT) k_member(const uint32_t *__restrict__ run_of,
                                               const uint32_t *__restrict__ parent,
                                               const uint32_t *__restrict__ cand_of_root,
                                               const uint32_t *__restrict__ cat_of_cand,
                                               const SPos<PT> *__restrict__ spos,
                                               const DevScal *__restrict__ sc,
                                               unsigned long long *__restrict__ member) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const int64_t np = sc->np;
  for (int64_t i = gtid(); i < np; i += gstride()) {
    const uint32_t ci = cand_of_root[parent[run_of[i]]];
    if (ci == kNone) continue;
    const uint32_t h = cat_of_cand[ci];
    if (h == kNone) continue;
    atomicMin(member + spos[i].src, (unsigned long long)h);
  }
}

template <class PT>
__global__ void __launch_bounds__(kT) k_member_copy(
    const uint32_t *__restrict__ run_of, const uint32_t *__restrict__ parent,
    const uint32_t *__restrict__ cand_of_root, const uint32_t *__restrict__ cat_of_cand,
    const uint16_t *__restrict__ run_box, const uint32_t *__restrict__ boxd, int nbox,
    const SPos<PT> *__restrict__ spos, const uint32_t *__restrict__ perm,
    const DevScal *__restrict__ sc, const unsigned long long *__restrict__ member,
    uint32_t *__restrict__ member_proc, float *__restrict__ member_pos, Counters *ctr) {
  if (sc->failed) return;  // a sort of this run gave up: its order is not valid
  const int64_t np = sc->np;
  for (int64_t i = gtid(); i < np; i += gstride()) {
    const uint32_t run = run_of[i];
    const uint32_t ci = cand_of_root[parent[run]];
    if (ci == kNone) continue;
    const uint32_t h = cat_of_cand[ci];
    if (h == kNone) continue;
    const SPos<PT> p = spos[i];
    if (member[p.src] == (unsigned long long)h) {
      if (!member_proc) continue;  // only the halo indices are wanted
      member_proc[p.src] = perm[i] - boxd[4 * nbox + run_box[run]];
      member_pos[3 * (uint64_t)p.src] = (float)p.x;
      member_pos[3 * (uint64_t)p.src + 1] = (float)p.y;
      member_pos[3 * (uint64_t)p.src + 2] = (float)p.z;
    } else {
      atomicAdd(&ctr->member_conflicts, 1ull);
    }
  }
}

int bits_for(uint64_t v) {
  int b = 0;
  while (b < 64 && (v >> b) != 0) b++;
  return b;
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------

namespace {
// Values of the position type in order as unsigned integers, and back.  (The
// ordinals of two doubles may be more than 2^63 apart.)
uint64_t ordinal(float x) {
  uint32_t i;
  memcpy(&i, &x, 4);
  return i >> 31 ? ~i : i | 0x80000000u;
}
uint64_t ordinal(double x) {
  uint64_t i;
  memcpy(&i, &x, 8);
  return i >> 63 ? ~i : i | 0x8000000000000000ull;
}
void from_ordinal(uint64_t o, float *x) {
  const uint32_t i = o >> 31 ? (uint32_t)o & 0x7fffffffu : ~(uint32_t)o;
  memcpy(x, &i, 4);
}
void from_ordinal(uint64_t o, double *x) {
  const uint64_t i = o >> 63 ? o & 0x7fffffffffffffffull : ~o;
  memcpy(x, &i, 8);
}

// The smallest (dir > 0) or largest (dir < 0) value x of the position type for
// which ok(x) holds, ok being monotonic with its bound within `slack` of
// `guess`; an infinity when it holds nowhere.
template <class PT, class F> PT edge_value(double guess, double slack, int dir, F ok) {
  const PT inf = std::numeric_limits<PT>::infinity();
  PT in = (PT)(guess + dir * slack), out = (PT)(guess - dir * slack);
  if (!ok(in)) in = dir * std::numeric_limits<PT>::max();
  if (!ok(in)) return dir * inf;
  if (ok(out)) out = -dir * inf;  // (no coordinate: ok() is not asked about it)
  uint64_t a = ordinal(in), b = ordinal(out);
  while ((a > b ? a - b : b - a) > 1) {
    const uint64_t m = a > b ? b + (a - b) / 2 : a + (b - a) / 2;
    PT x;
    from_ordinal(m, &x);
    if (ok(x)) a = m;
    else b = m;
  }
  PT x;
  from_ordinal(a, &x);
  return x;
}

// The ingest's thresholds along an axis (see Geom).
template <class PT> void ingest_thresholds(Geom &g, int a) {
  const double lo = g.periodic ? g.lo[a] : g.rmin[a], hi = g.periodic ? g.hi[a] : g.rmax[a];
  const double slack = 4.0 * (double)std::numeric_limits<PT>::epsilon() *
                       (std::fabs(g.rmin[a]) + std::fabs(g.rmax[a]) + g.L[a]);
  g.dom_lo[a] = (double)edge_value<PT>(lo, slack, 1, [&](PT x) { return (double)x >= lo; });
  g.dom_hi[a] = (double)edge_value<PT>(hi, slack, -1, [&](PT x) { return (double)x <= hi; });
  g.img_lo[a] = std::numeric_limits<double>::infinity();
  g.img_hi[a] = -std::numeric_limits<double>::infinity();
  if (!g.periodic) return;
  // (an image by -L lies below hi, one by +L above lo, whatever the rounding)
  g.img_lo[a] = (double)edge_value<PT>(g.rmin[a] + g.L[a], slack, 1, [&](PT x) {
    return (double)(PT)((double)x - g.L[a]) >= g.rmin[a];
  });
  g.img_hi[a] = (double)edge_value<PT>(g.rmax[a] - g.L[a], slack, -1, [&](PT x) {
    return (double)(PT)((double)x + g.L[a]) <= g.rmax[a];
  });
}
}  // namespace

Geom Plan::make_geometry(const cmh_fof_params &p, const std::vector<double> &ltab,
                         int64_t n_in, int cell_factor) const {
  Geom g{};
  double minlink = p.linklength, maxlink = p.linklength;
  if (p.varlink) {
    minlink = maxlink = ltab.empty() ? p.linklength : ltab[0];
    for (double v : ltab) {
      minlink = std::min(minlink, v);
      maxlink = std::max(maxlink, v);
    }
  }
  if (!(minlink > 0) || !std::isfinite(maxlink))
    fail(CMH_ERR_INVALID_ARGUMENT, "linking length must be positive and finite");
  for (int a = 0; a < 3; a++) {
    g.lo[a] = p.lo[a];
    g.hi[a] = p.hi[a];
    g.rmin[a] = p.lo[a] - p.boundary;  // startup.c:40-47
    g.rmax[a] = p.hi[a] + p.boundary;
    g.L[a] = p.hi[a] - p.lo[a];
    if (!(g.L[a] > 0)) fail(CMH_ERR_INVALID_ARGUMENT, "box extent must be positive");
  }
  g.boundary = p.boundary;
  g.linksq = p.linklength * p.linklength;  // FOF.c:60
  g.maxlink = maxlink;
  g.prune_sq = (maxlink * (1.0 + 1e-5)) * (maxlink * (1.0 + 1e-5));
  g.nphalomin = p.nphalomin;
  g.periodic = p.periodic ? 1 : 0;
  g.props = (int)(p.properties & 3u);
  g.hs = 7 + ((g.props & 1) ? 6 : 0) + ((g.props & 2) ? 6 : 0);
  band_thresholds(g.linksq, pos_dtype == CMH_FLOAT64 ? 8 : 4, &g.t_lo, &g.t_hi);
  // fine cell: any two points of a cell are closer than minlink
  g.h = minlink * (1.0 - 0x1p-20) / std::sqrt(3.0);
  g.inv_h = 1.0 / g.h;
  g.W = (int)std::floor(maxlink / g.h * (1.0 + 1e-6)) + 1;
  if (p.varlink) {
    // the fixed grid of the l(r) rule (FOF.c:50-52, 63-65)
    g.varlink = 1;
    for (int a = 0; a < 3; a++) {
      if (p.ref_cells[a] < 1) fail(CMH_ERR_INVALID_ARGUMENT, "ref_cells must be positive");
      g.origin[a] = p.origin[a];
      g.ref_lcell[a] = (p.hi[a] - p.lo[a] + 2.0 * p.boundary) / p.ref_cells[a];
      g.ref_nc[a] = (int)std::ceil((g.rmax[a] - g.rmin[a]) / g.ref_lcell[a]) + 1;
      if (g.ref_nc[a] >= (1 << 21)) fail(CMH_ERR_CAPACITY, "more than 2^21 grid cells along an axis");
      // the reference scans only neighbouring cells: a longer link would be missed
      if (maxlink > g.ref_lcell[a])
        fail(CMH_ERR_INVALID_ARGUMENT, "linking length longer than the grid cell (raise Px/Py/Pz cells)");
    }
    if (ltab.size() < 2 || !(p.ltab_rmax > 0))
      fail(CMH_ERR_INVALID_ARGUMENT, "variable linking length needs a table of 2+ values");
    g.ltab_n = (int)ltab.size();
    g.ltab_dr = p.ltab_rmax / (double)(g.ltab_n - 1);
  }
  for (int a = 0; a < 3; a++) {
    if (pos_dtype == CMH_FLOAT64) ingest_thresholds<double>(g, a);
    else ingest_thresholds<float>(g, a);
  }
  double vol = 1.0;
  for (int a = 0; a < 3; a++) {
    g.G[a] = (int)std::floor((g.rmax[a] - g.rmin[a]) / g.h) + 2;
    if (g.G[a] >= (1 << 21)) fail(CMH_ERR_CAPACITY, "more than 2^21 fine cells along an axis");
    vol *= (g.rmax[a] - g.rmin[a]);
  }
  int k = cell_factor > 0 ? cell_factor : p.cell_factor;
  if (k <= 0) {
    // About one top cell per particle, as the reference's lcell = L/Px, or the
    // tuned scale of it.  Untuned, somewhat smaller top cells for runs of up to
    // 32M particles, where the largest dense top cells bound the befriending
    // (scale 0.85 against 1: 64^3 box 0.361 and 0.384 ms, 1.5M particles 0.67 and
    // 0.71, 64 boxes 10.5 and 10.9, 256^3 box 3.43 and 3.43, but the 512^3 box 32.9
    // and 32.4; the line lies between the last two, with no size measured between);
    // and none of more than 10^3 fine cells where that leaves at
    // most four top cells per particle (50M lightcone 10.6 ms with 10, 11.5 with
    // 14; 700,000-particle one 0.57 and 0.73), in runs whose top-cell tables are
    // small beside the device's memory.
    const double sep = std::cbrt(vol / std::max<double>((double)n_in, 1.0)) / g.h;
    if (cell_scale > 0) {
      k = (int)std::lround(sep * cell_scale);
    } else {
      k = (int)std::lround(sep * (n_in <= (int64_t)1 << 25 ? 0.85 : 1.0));
      if (n_in < (int64_t)1 << 28) k = std::min(k, std::max(10, (int)std::ceil(0.63 * sep)));
    }
  }
  if (g.W > kMaxCellFactor)
    fail(CMH_ERR_INVALID_ARGUMENT, "linking lengths span too wide a range (longest / shortest "
                                   "above 18): a fine cell's reach would leave the 27 top cells");
  k = std::min(std::max(k, g.W), kMaxCellFactor);
  while (true) {
    uint64_t T = 1;
    for (int a = 0; a < 3; a++) {
      g.T[a] = (g.G[a] + k - 1) / k;
      T *= (uint64_t)g.T[a];
    }
    if (T < (1ull << 31) || k >= kMaxCellFactor) {
      if (T >= (1ull << 31)) fail(CMH_ERR_CAPACITY, "domain too large for the top-cell grid");
      g.k = k;
      g.k3 = (uint64_t)k * k * k;
      g.kmul = (uint32_t)((1ull << 32) / (uint64_t)k + 1);
      break;
    }
    k++;
  }
  return g;
}

namespace {
// Grid of a grid-stride kernel of kT threads: the CTAs that can be resident
// at once, capped by the work.
template <class K> unsigned rg(K *kernel, int64_t n) {
  return grid_resident(reinterpret_cast<const void *>(kernel), kT, 0, n);
}

// Shared-memory words of one dense top cell: k^3 parents, k^2 bit rows, k^2
// row prefixes, k^2 rows of the cells outside the main component, the count of
// components and the main one's root.
uint64_t dense_words(uint64_t k3all) {
  const uint64_t k = (uint64_t)std::llround(std::cbrt((double)k3all));
  return k3all + 3 * k * k + 2;
}

// Fine cells above which a dense top cell is joined by a whole CTA, not a warp.
// A CTA shortens one top cell's chain of steps, which bounds a small run, but
// waits at its barriers, which costs a large one.  Befriending with 32, 64, 128
// and 300: 64^3 box 0.137, 0.150, 0.187, 0.215 ms; 1.5M particles 0.231, 0.223,
// 0.262, 0.332; 256^3 box 1.16, 1.11, 1.09, 1.14; 512^3 box 14.3, 13.1, 12.5, 12.1.
// The power law passes near the best of these four.
uint32_t big_top_min(int64_t np) {
  return (uint32_t)std::max(32.0, 48.0 * std::pow((double)np / 1e6, 0.35));
}

// Warps per CTA of the dense-top kernel: up to 4, each with the words of one
// top cell, within 200 KiB per CTA.
int dense_warps_per_cta(uint64_t k3all) {
  const uint64_t per = dense_words(k3all) * sizeof(uint32_t);
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(4, (200u << 10) / per));
}

// 16-byte words of a dense top cell's occupancy: planes, then k^2 rows.
uint64_t rows_per_top(uint64_t k3all) {
  const uint64_t k = (uint64_t)std::llround(std::cbrt((double)k3all));
  return row_head((int)k) + k * k;
}

// Dense top cells whose planes and rows fit in 4 bytes per processed
// particle plus 1 GiB.
int64_t rows_cap_for(int64_t np_cap, uint64_t k3all) {
  return (int64_t)(((uint64_t)np_cap * 4 + (1ull << 30)) / (rows_per_top(k3all) * sizeof(uint4)));
}

// The dense-top kernel's limit of dynamic shared memory belongs to the kernel and
// device, not to a launch: while runs of several plans overlap (from several
// threads) it is the most that one of them takes.  (The largest possible at all
// times makes the driver give the SMs less L1: 256^3 box 3.24 -> 3.30 ms, 50M
// lightcone 10.1 -> 10.3.)  `bytes`: what the plan's run takes; 0 when it has ended.
void dense_room(const Plan *plan, int device, int bytes) {
  struct Needs {
    std::mutex mu;
    std::map<std::pair<int, const Plan *>, int> of;
  };
  static Needs *needs = new Needs;  // (never freed: a run may outlive static objects)
  std::lock_guard<std::mutex> lock(needs->mu);
  if (bytes == 0) {
    needs->of.erase({device, plan});
    return;
  }
  needs->of[{device, plan}] = bytes;
  int most = 0;
  for (const auto &q : needs->of)
    if (q.first.first == device) most = std::max(most, q.second);
  const void *dense[] = {
      (const void *)k_befriend_dense<float, true, false>,
      (const void *)k_befriend_dense<float, false, false>,
      (const void *)k_befriend_dense<double, true, false>,
      (const void *)k_befriend_dense<double, false, false>,
      (const void *)k_befriend_dense<float, true, true>,
      (const void *)k_befriend_dense<float, false, true>,
      (const void *)k_befriend_dense<double, true, true>,
      (const void *)k_befriend_dense<double, false, true>};
  for (const void *f : dense)
    CMH_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CMH_CUDA(cudaStreamIsCapturing(s, &cs));
  return cs == cudaStreamCaptureStatusActive;
}

// An event record that other streams can wait on also when it is replayed
// from a recorded graph.
void record_external(cudaEvent_t e, cudaStream_t s) {
  if (capturing(s)) CMH_CUDA(cudaEventRecordWithFlags(e, s, cudaEventRecordExternal));
  else CMH_CUDA(cudaEventRecord(e, s));
}

// Bytes of a bucket's records: one fits in L2 (126 MB) beside the rest of what the
// gather touches.  8, 16, 32 and 64 MB: gather of the 512^3 box 6.2 to 6.4 ms
// with its scans, but its ingest 4.7, 4.7, 4.4 and 4.0 ms (fewer places to take
// per tile, longer runs to write).
constexpr double kBucketBytes = 64e6;

// Images per input particle expected for a periodic box (the shell's share
// of the padded volume), with headroom for clustering.
double image_estimate(const Geom &g, int64_t n) {
  if (!g.periodic) return 0.0;
  double f = 1.0;
  for (int a = 0; a < 3; a++) f *= (g.L[a] + 2 * g.boundary) / g.L[a];
  return (double)n * (f - 1.0) * 1.5 + 4096.0;
}
}  // namespace

template <class PT>
void Plan::issue(int want_member, cudaStream_t s, bool timed) {
  const int nbox = (int)boxes_host.size();
  const int64_t n = n_total, npc = np_cap, ncc = nc_cap;
  DevScal *sc = scal.as<DevScal>();
  unsigned char *small = scal.as<unsigned char>();
  Counters *c = reinterpret_cast<Counters *>(small + at_ctr);
  unsigned long long *extra = reinterpret_cast<unsigned long long *>(c + 1);  // ngroups, nwarn
  uint32_t *boxd = reinterpret_cast<uint32_t *>(small + at_boxd);
  uint32_t *bucket = reinterpret_cast<uint32_t *>(small + at_bucket);
  uint32_t *cell_counts = reinterpret_cast<uint32_t *>(small + at_counts);
  const BoxDev *boxes = b_boxes.as<BoxDev>();
  // buffers whose lifetimes do not overlap share memory: the fine-cell tables
  // lie in the sort's keys, dead after its last pass, and the befriending queue
  // in the records, dead after the gather
  uint64_t *run_g = b_keys.as<uint64_t>();
  uint32_t *run_of = b_keys_alt.as<uint32_t>(), *run_start = run_of + npc;  // npc + 1
  uint32_t *parent = b_parent.as<uint32_t>();
  uint32_t *q_cell = b_recs.as<uint32_t>(), *q_top = q_cell + npc;
  uint2 *tile_sum = b_tiles.as<uint2>();
  auto mark = [&](int q) {
    if (timed) CMH_CUDA(cudaEventRecord(q < 0 ? ev0 : (q >= 7 ? ev1 : stage_ev[q]), s));
  };
  mark(-1);
  // the run's scalars, counters, per-box numbers, buckets and digit counts
  CMH_CUDA(cudaMemsetAsync(scal.p, 0, small_bytes, s));

  // ---- ingest ----
  // beside it, on the second stream, the clearing of the later stages' tables
  // (their first users wait for it)
  const int NS = 6 + ((props & 1) ? 6 : 0) + ((props & 2) ? 6 : 0);
  CMH_CUDA(cudaEventRecord(ev_fork, s));
  CMH_CUDA(cudaStreamWaitEvent(bf_stream, ev_fork, 0));
  {
    Fills f;
    f.add(b_top_range, n_top * 8, 0u);
    f.add(b_top_slot, n_top * 4, 0xffffffffu);
    f.add(b_cand_of_root, npc * 4, 0xffffffffu);
    f.add(b_sums, (size_t)ncc * NS * 8, 0u);
    f.add(b_warn, (size_t)ncc * 4, 0u);
    f.add(b_cat_of_cand, (size_t)ncc * 4, 0xffffffffu);
    f.add(b_count, npc * 4, 0u);
    f.add(b_head, (size_t)ncc * 4, 0xffffffffu);
    f.add(b_marks, (size_t)((npc + kHeadGroup - 1) / kHeadGroup) * (kHeadGroup / 8), 0u);
    f.add(b_run_state, (size_t)run_tiles * 8, 0u);
    if (cell_states_apart) f.add(sort_tmp, cell_state_bytes, 0u);
    if (want_member && n > 0) {
      f.add(b_member, (size_t)n * 8, 0xffffffffu);
      if (want_member == 1) {
        f.add(b_member_proc, (size_t)n * 4, 0xffffffffu);
        f.add(b_member_pos, (size_t)n * 12, 0u);
      }
    }
    uint64_t most = 0;
    for (int q = 0; q < f.count; q++) most = std::max(most, f.n[q]);
    k_fill<<<grid_for((int64_t)most, kT, 4), kT, 0, bf_stream>>>(f);
    CMH_LAUNCHED();
  }
  CMH_CUDA(cudaEventRecord(ev_cleared, bf_stream));
  const PassDigits pd = radix_order_plan(key_bits);
  const size_t hist_smem = (size_t)pd.passes * kRadixBins * 4;
  auto ingest = [&](auto per) {
    constexpr int PER = decltype(per)::value;
    if (n > 0) {
      k_ingest_count<PT, PER><<<rg(k_ingest_count<PT, PER>, (int64_t)n_tiles * kT), kT, 0, s>>>(
          boxes, nbox, n_tiles, n_buckets, tile_sum, bucket);
      CMH_LAUNCHED();
    }
    k_ingest_scan<<<1, kScanT, 0, s>>>(boxes, nbox, n_tiles, n_buckets, tile_sum, bucket, sc, boxd,
                                       (uint32_t)npc);
    CMH_LAUNCHED();
    if (n > 0) {
      k_ingest_emit<PT, PER><<<grid_resident((const void *)k_ingest_emit<PT, PER>, kT, hist_smem,
                                             (int64_t)n_tiles * kT),
                               kT, hist_smem, s>>>(
          boxes, nbox, n_tiles, n_buckets, k3all, tile_sum, bucket, boxd, (uint32_t)npc,
          b_recs.as<PRec<PT>>(), pd, cell_counts);
      CMH_LAUNCHED();
    }
  };
  if (ingest_per == kPer) ingest(std::integral_constant<int, kPer>{});
  else ingest(std::integral_constant<int, 1>{});
  mark(0);
  // host inputs: their positions are read no more (a next run's may be
  // copied into their buffer)
  if (vel_wait) record_external(ev_pos_free, s);
  // ---- sort ----
  // the sort leaves the records' indices in cell order and no sorted keys;
  // a look-back that gives up raises sc->failed, and every later kernel of
  // the run then returns at once (the order would not be valid)
  const bool odd = pd.passes % 2 == 1;
  uint32_t *order = odd ? b_vals_alt.as<uint32_t>() : b_vals.as<uint32_t>();
  uint32_t *perm = odd ? b_vals.as<uint32_t>() : b_vals_alt.as<uint32_t>();
  if (cell_states_apart) CMH_CUDA(cudaStreamWaitEvent(s, ev_cleared, 0));
  radix_order_records(b_recs.p, sizeof(PRec<PT>), offsetof(PRec<PT>, key), b_keys.as<uint64_t>(),
                      b_vals.as<uint32_t>(), b_keys_alt.as<uint64_t>(), b_vals_alt.as<uint32_t>(),
                      npc, &sc->np, key_bits,
                      RadixTmp{sort_tmp.as<uint64_t>(), cell_counts, cell_states_apart},
                      &sc->failed, s, SortWaits{spin_cap, stall_sort ? 1u : 0xffffffffu});
  mark(1);
  // ---- runs, top-cell ranges, dense top cells ----
  CMH_CUDA(cudaStreamWaitEvent(s, ev_cleared, 0));  // the later stages' tables
  auto gather = [&](auto per) {
    k_gather_runs<PT, decltype(per)::value><<<(unsigned)run_tiles, kT, 0, s>>>(
        order, b_recs.as<PRec<PT>>(), boxes, nbox, b_spos.as<SPos<PT>>(), perm, run_of, run_start,
        run_g, b_run_box.as<uint16_t>(), parent, b_top_range.as<uint32_t>(),
        b_run_state.as<uint64_t>(), sc, SortWaits{spin_cap, stall_gather ? 1u : 0xffffffffu});
    CMH_LAUNCHED();
  };
  if (run_per == kRunPerLarge) gather(std::integral_constant<int, kRunPerLarge>{});
  else gather(std::integral_constant<int, kRunPerSmall>{});
  if (varlink) {
    if (fp32)
      k_varlink_recs<PT, true><<<rg(k_varlink_recs<PT, true>, npc), kT, 0, s>>>(b_spos.as<SPos<PT>>(), run_of,
                                                 b_run_box.as<uint16_t>(), boxes, sc,
                                                 b_svl.as<VLRec64>());
    else
      k_varlink_recs<PT, false><<<rg(k_varlink_recs<PT, false>, npc), kT, 0, s>>>(b_spos.as<SPos<PT>>(), run_of,
                                                  b_run_box.as<uint16_t>(), boxes, sc,
                                                  b_svl.as<VLRec64>());
    CMH_LAUNCHED();
  }
  const uint32_t big_min = big_top_min(npc);
  k_dense_pick<<<rg(k_dense_pick, npc), kT, 0, s>>>(
      run_g, b_run_box.as<uint16_t>(), boxes, sc, b_top_range.as<uint2>(), dense_min, big_min,
      (uint32_t)nd_cap, b_top_slot.as<uint32_t>(), b_dense_range.as<uint2>(),
      b_dense_big.as<uint32_t>());
  CMH_LAUNCHED();
  mark(2);
  // ---- befriending: dense top cells inside (CTA each) on a second stream
  // while the sparse path runs (both join cells through the lock-free
  // union-find), then the queued items of dense neighbours, near then far ----
  const uint32_t q_cap = (uint32_t)npc;
  const int dwpc = dense_warps_per_cta(k3all);
  const uint32_t kmax = (uint32_t)std::llround(std::cbrt((double)k3all)), kk = kmax * kmax;
  const uint32_t rows_stride = (uint32_t)rows_per_top(k3all);
  const size_t dsm = (size_t)dwpc * dense_words(k3all) * sizeof(uint32_t);
  const unsigned gd = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>((nd_cap + dwpc - 1) / dwpc, (int64_t)kSMs * 64 / dwpc));
  auto befriend = [&](auto fp32_tag, auto vl_tag) {
    constexpr bool FP = decltype(fp32_tag)::value;
    constexpr bool VL = decltype(vl_tag)::value;
    const VLRec<FP> *svl = VL ? b_svl.as<VLRec<FP>>() : nullptr;
    // dense top cells on a second stream, beside the sparse cells
    CMH_CUDA(cudaEventRecord(ev_fork, s));
    CMH_CUDA(cudaStreamWaitEvent(bf_stream, ev_fork, 0));
    const PairArgs<PT, FP> pa{boxes, b_run_box.as<uint16_t>(), run_start, run_g,
                              b_spos.as<SPos<PT>>(), svl, c};
    k_befriend_dense<PT, FP, VL><<<gd, 32 * dwpc, dsm, bf_stream>>>(
        pa, k3all, b_dense_range.as<uint2>(), b_dense_big.as<uint32_t>(), sc, (uint32_t)nd_cap,
        b_rows.as<uint4>(), kk, rows_stride, parent, (uint32_t)dense_words(k3all),
        big_min);
    CMH_LAUNCHED();
    CMH_CUDA(cudaEventRecord(ev_join, bf_stream));
    k_befriend_sparse<PT, FP, VL><<<rg(k_befriend_sparse<PT, FP, VL>, npc), kT, 0, s>>>(
        pa, sc, b_top_range.as<uint2>(), b_top_slot.as<uint32_t>(), parent,
        q_cell, q_top, q_cap, dense_min);
    CMH_LAUNCHED();
    CMH_CUDA(cudaStreamWaitEvent(s, ev_join, 0));
    k_befriend_cross<PT, FP, VL, 0><<<rg(k_befriend_cross<PT, FP, VL, 0>, npc * 8), kT, 0, s>>>(
        pa, q_cell, q_top, q_cap, sc, b_rows.as<uint4>(), rows_stride, parent);
    CMH_LAUNCHED();
    k_compress<<<rg(k_compress, npc), kT, 0, s>>>(parent, sc);
    CMH_LAUNCHED();
    k_befriend_cross<PT, FP, VL, 1><<<rg(k_befriend_cross<PT, FP, VL, 1>, npc * 8), kT, 0, s>>>(
        pa, q_cell, q_top, q_cap, sc, b_rows.as<uint4>(), rows_stride, parent);
    CMH_LAUNCHED();
  };
  if (fp32 && varlink) befriend(std::true_type{}, std::true_type{});
  else if (fp32) befriend(std::true_type{}, std::false_type{});
  else if (varlink) befriend(std::false_type{}, std::true_type{});
  else befriend(std::false_type{}, std::false_type{});
  mark(3);

  // ---- groups, candidates ----
  k_compress_count<<<rg(k_compress_count, npc), kT, 0, s>>>(parent, run_start, sc,
                                                            b_count.as<uint32_t>());
  CMH_LAUNCHED();
  if (sampling && n > 0) {
    CMH_CUDA(cudaMemsetAsync(b_samp.p, 0, (size_t)n, s));
    k_subsample<PT><<<rg(k_subsample<PT>, npc), kT, 0, s>>>(
        run_of, parent, b_count.as<uint32_t>(), perm,
        b_spos.as<SPos<PT>>(), b_run_box.as<uint16_t>(), boxes, boxd, nbox, sc, samp_ids,
        samp_in, samp_out, samp_seed, samp_closed, b_samp.as<uint8_t>());
    CMH_LAUNCHED();
  }
  k_cand_pick<<<rg(k_cand_pick, npc), kT, 0, s>>>(
      parent, b_count.as<uint32_t>(), b_run_box.as<uint16_t>(), boxes, sc,
      b_cand_of_root.as<uint32_t>(), b_cand_root.as<uint32_t>(), extra + 0);
  CMH_LAUNCHED();
  mark(4);

  // ---- property sums, ownership, catalog ----
  if (vel_wait) {
    // host-resident velocities arrive on the side stream while the steps
    // above run; the sums are their first reader
    CMH_CUDA(cudaStreamWaitEvent(s, ev_vel_ready,
                                 capturing(s) ? cudaEventWaitExternal : cudaEventWaitDefault));
  }
#define CMH_SUMS(NSV)                                                                         \
  k_group_sums<PT, NSV><<<rg(k_group_sums<PT, NSV>, npc), kT, 0, s>>>(run_of, parent,  \
                                          b_cand_of_root.as<uint32_t>(),                      \
                                          b_run_box.as<uint16_t>(), boxes,                    \
                                          b_spos.as<SPos<PT>>(), perm, sc, props,             \
                                          b_sums.as<double>(), b_head.as<uint32_t>(),         \
                                          b_warn.as<uint32_t>())
  if (NS == 6) CMH_SUMS(6);
  else if (NS == 12) CMH_SUMS(12);
  else CMH_SUMS(18);
#undef CMH_SUMS
  CMH_LAUNCHED();
  mark(5);
  if (vel_wait) record_external(ev_vel_free, s);  // nor their velocities
  const uint32_t ngroup = (uint32_t)((npc + kHeadGroup - 1) / kHeadGroup);
  uint32_t *marks = b_marks.as<uint32_t>(), *group = marks + (size_t)ngroup * 32;
#define CMH_OWNED(NSV)                                                                          \
  k_own_pick<NSV><<<rg(k_own_pick<NSV>, ncc), kT, 0, s>>>(                                      \
      b_sums.as<double>(), b_cand_root.as<uint32_t>(), b_count.as<uint32_t>(),                  \
      b_head.as<uint32_t>(), b_run_box.as<uint16_t>(), boxes, sc, b_own_head.as<uint32_t>(),    \
      b_own_cand.as<uint32_t>(), marks, (uint32_t)npc, boxd, nbox)
  if (NS == 6) CMH_OWNED(6);
  else if (NS == 12) CMH_OWNED(12);
  else CMH_OWNED(18);
#undef CMH_OWNED
  CMH_LAUNCHED();
  k_head_groups<<<rg(k_head_groups, (int64_t)ngroup * 32), kT, 0, s>>>(marks, ngroup, group, sc);
  CMH_LAUNCHED();
  k_head_scan<<<1, kScanT, 0, s>>>(group, ngroup, boxd, nbox, sc);
  CMH_LAUNCHED();
#define CMH_CATALOG(NSV)                                                                        \
  k_catalog<NSV><<<rg(k_catalog<NSV>, ncc), kT, 0, s>>>(b_own_head.as<uint32_t>(),             \
                                   b_own_cand.as<uint32_t>(), marks, group, sc,                  \
                                   b_sums.as<double>(), b_cand_root.as<uint32_t>(),             \
                                   b_count.as<uint32_t>(), b_warn.as<uint32_t>(),               \
                                   b_run_box.as<uint16_t>(), boxd, nbox, props, hs,              \
                                   b_props.as<float>(), b_head_out.as<uint32_t>(),              \
                                   b_cat_of_cand.as<uint32_t>(), extra + 1)
  if (NS == 6) CMH_CATALOG(6);
  else if (NS == 12) CMH_CATALOG(12);
  else CMH_CATALOG(18);
#undef CMH_CATALOG
  CMH_LAUNCHED();
  mark(6);
  if (want_member && n > 0) {
    k_member<PT><<<rg(k_member<PT>, npc), kT, 0, s>>>(run_of, parent,
                                   b_cand_of_root.as<uint32_t>(), b_cat_of_cand.as<uint32_t>(),
                                   b_spos.as<SPos<PT>>(), sc, b_member.as<unsigned long long>());
    CMH_LAUNCHED();
    k_member_copy<PT><<<rg(k_member_copy<PT>, npc), kT, 0, s>>>(
        run_of, parent, b_cand_of_root.as<uint32_t>(),
        b_cat_of_cand.as<uint32_t>(), b_run_box.as<uint16_t>(), boxd, nbox,
        b_spos.as<SPos<PT>>(), perm, sc, b_member.as<unsigned long long>(),
        b_member_proc.as<uint32_t>(), b_member_pos.as<float>(), c);
    CMH_LAUNCHED();
  }
  mark(7);
}

void Plan::prepare(const std::vector<BoxSpec> &specs, int want_member) {
  if (!bf_stream) {
    CMH_CUDA(cudaStreamCreateWithFlags(&bf_stream, cudaStreamNonBlocking));
    CMH_CUDA(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
    CMH_CUDA(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
    CMH_CUDA(cudaEventCreateWithFlags(&ev_cleared, cudaEventDisableTiming));
  }
  const int nbox = (int)specs.size();
  if (nbox < 1 || nbox > kMaxBoxes) fail(CMH_ERR_INVALID_ARGUMENT, "1 to 1024 boxes per run");
  boxes_host.resize(nbox);
  n_total = 0;
  for (const BoxSpec &sp : specs) n_total += sp.n;
  ingest_per = n_total >= (int64_t)kSMs * 4 * kT * kPer ? kPer : 1;
  n_total = 0;
  n_tiles = 0;
  uint64_t tops = 0;
  int kmax = 1;
  double img = 0.0;
  props = -1;
  for (int b = 0; b < nbox; b++) {
    const BoxSpec &sp = specs[b];
    BoxDev &bd = boxes_host[b];
    memset(&bd, 0, sizeof bd);
    bd.g = make_geometry(sp.params, sp.ltab, sp.n, sp.cell_factor);
    bd.g.union_cap = union_cap;
    if (props < 0) props = bd.g.props;
    if (bd.g.props != props) fail(CMH_ERR_INVALID_ARGUMENT, "boxes of a run share the property set");
    bd.pos = sp.pos;
    bd.vel = sp.vel;
    bd.vel_f64 = sp.vel_f64 ? 1 : 0;
    bd.n = (uint32_t)sp.n;
    bd.in_base = (uint64_t)n_total;
    bd.top_base = tops;
    bd.tile_base = n_tiles;
    n_tiles += (uint32_t)((sp.n + kT * ingest_per - 1) / (kT * ingest_per));
    n_total += sp.n;
    tops += (uint64_t)bd.g.T[0] * bd.g.T[1] * bd.g.T[2];
    kmax = std::max(kmax, bd.g.k);
    img += image_estimate(bd.g, sp.n);
  }
  if (n_total >= (int64_t)0xfffffff0ll) fail(CMH_ERR_CAPACITY, "more than 2^32 input particles in a run");
  // buckets of the emission: slabs whose records take about kBucketBytes, at
  // least one per box
  {
    const size_t rec = pos_dtype == CMH_FLOAT64 ? sizeof(PRec<double>) : sizeof(PRec<float>);
    const double want =
        std::min(512.0, std::ceil(((double)n_total + img) * (double)rec / kBucketBytes));
    n_buckets = 0;
    for (int b = 0; b < nbox; b++) {
      BoxDev &bd = boxes_host[b];
      const double share = n_total > 0 ? (double)bd.n / (double)n_total : 1.0;
      bd.bucket_base = (uint32_t)n_buckets;
      bd.nbucket = (uint32_t)std::max(1, (int)(want * share));
      bd.bucket_scale = (float)((double)bd.nbucket / (bd.g.rmax[2] - bd.g.rmin[2]));
      n_buckets += (int)bd.nbucket;
    }
  }
  // linking-length tables of all boxes, one device array
  varlink = false;
  ltab_all.clear();
  for (int b = 0; b < nbox; b++)
    if (boxes_host[b].g.varlink) {
      varlink = true;
      ltab_all.insert(ltab_all.end(), specs[b].ltab.begin(), specs[b].ltab.end());
    }
  if (varlink) {
    if (ltab_all.size() * sizeof(double) > ltab_dev.cap) uploaded_sig.clear();
    ltab_dev.ensure(ltab_all.size() * sizeof(double));
    size_t off = 0;
    for (int b = 0; b < nbox; b++)
      if (boxes_host[b].g.varlink) {
        boxes_host[b].g.ltab = ltab_dev.as<double>() + off;
        off += specs[b].ltab.size();
      }
  }
  hs = 7 + ((props & 1) ? 6 : 0) + ((props & 2) ? 6 : 0);
  k3all = (uint64_t)kmax * kmax * kmax;
  n_top = tops;
  key_bits = bits_for(tops * k3all - 1);
  if (tops >= (1ull << 40) || key_bits > 62) fail(CMH_ERR_CAPACITY, "too many cells in a run");
  // capacities: grown after a run that overflowed them, never shrunk
  const int64_t want_np = std::min<int64_t>(n_total + (int64_t)img, (int64_t)0xfffffff0ll);
  np_cap = std::max<int64_t>(np_cap, std::max<int64_t>(want_np, 1));
  // dense top cells: their rows take at most 4 bytes per processed particle
  // plus 1 GiB (dense top cells past the cap are scanned instead)
  // (a first run that finds more of them than slots scans the rest, ~3x the
  // befriending time: the 1024^3 workload's parameters have one dense top cell
  // per 650 processed particles, the 256^3 ones one per 1100)
  nd_cap = std::max<int64_t>(nd_cap, std::max(np_cap / 1024 + 1024, np_cap / 256));
  nd_cap = std::min<int64_t>(nd_cap, std::max<int64_t>(1024, rows_cap_for(np_cap, k3all)));
  double mincut = 1e18;
  for (const BoxDev &bd : boxes_host)  // (below 1, and NaN: every group is a candidate)
    mincut = std::min(mincut, bd.g.nphalomin >= 1.0 ? bd.g.nphalomin : 1.0);
  const int64_t div = (int64_t)std::floor(mincut);
  nc_cap = std::max<int64_t>(1, np_cap / div + 1);

  const int64_t nn = std::max<int64_t>(n_total, 1), npc = np_cap, ncc = nc_cap;
  // the run's buffers, laid out in one allocation (one cudaMalloc and cudaFree
  // where each buffer had its own: a one-shot run spent most of its time there)
  std::vector<std::pair<DevBuf *, size_t>> pieces;
  auto need = [&](DevBuf &b, size_t bytes) { pieces.emplace_back(&b, bytes); };
  // the small arrays that every run starts cleared, in one piece; the first
  // three are read back together
  auto up = [](size_t b) { return (b + 127) & ~(size_t)127; };
  at_ctr = up(sizeof(DevScal));
  at_boxd = at_ctr + up(sizeof(Counters) + 2 * sizeof(unsigned long long));
  at_bucket = at_boxd + up(sizeof(uint32_t) * 7 * nbox);
  at_counts = at_bucket + up((size_t)n_buckets * 4);
  small_bytes = at_counts + kRadixCounts * 4;
  need(scal, small_bytes);
  need(b_boxes, sizeof(BoxDev) * nbox);
  need(b_keys, npc * 8);
  need(b_keys_alt, npc * 8 + 8);  // (also run_of and run_start)
  need(b_parent, npc * 4);
  run_per = npc >= (int64_t)kSMs * 4 * kT * kRunPerLarge ? kRunPerLarge : kRunPerSmall;
  run_tiles = (npc + kT * run_per - 1) / (kT * run_per);
  need(b_run_state, (size_t)run_tiles * 8);
  need(b_vals, npc * 4);
  need(b_vals_alt, npc * 4);
  const bool dbl = pos_dtype == CMH_FLOAT64;
  need(b_recs, npc * (dbl ? sizeof(PRec<double>) : sizeof(PRec<float>)));
  need(b_spos, npc * (dbl ? sizeof(SPos<double>) : sizeof(SPos<float>)));
  need(b_tiles, (size_t)n_tiles * sizeof(uint2));
  if (varlink) need(b_svl, npc * sizeof(VLRec64));
  need(b_run_box, npc * 2);
  need(b_top_range, n_top * 8);
  need(b_top_slot, n_top * 4);
  need(b_rows, (size_t)nd_cap * rows_per_top(k3all) * sizeof(uint4));
  need(b_dense_range, (size_t)nd_cap * sizeof(uint2));
  need(b_dense_big, (size_t)nd_cap * sizeof(uint32_t));
  need(b_count, npc * 4);
  need(b_head, ncc * 4);
  need(b_cand_of_root, npc * 4);
  if (sampling) need(b_samp, (size_t)nn);
  need(b_cand_root, ncc * 4);
  need(b_sums, ncc * 18 * 8);
  need(b_warn, ncc * 4);
  need(b_own_head, ncc * 4);
  need(b_own_cand, ncc * 4);
  // marks of the heads (a bit each) and the counts of their groups
  need(b_marks, (size_t)((npc + kHeadGroup - 1) / kHeadGroup) * (kHeadGroup / 8 + 4));
  need(b_props, ncc * hs * 4);
  need(b_head_out, ncc * 4);
  need(b_cat_of_cand, ncc * 4);
  if (want_member) need(b_member, nn * 8);
  if (want_member == 1) {
    need(b_member_proc, nn * 4);
    need(b_member_pos, nn * 12);
  }
  // shared memory of the dense-top kernel: one parent per fine cell of a top
  // cell (set here, outside any graph capture, until the run ends)
  dense_room(this, device,
             (int)(dense_warps_per_cta(k3all) * dense_words(k3all) * sizeof(uint32_t)));
  cell_states_apart = radix_states_apart(npc, key_bits, &cell_state_bytes);
  need(sort_tmp, cell_state_bytes);
  // (issue() allocates nothing: it may be captured in a graph)
  auto room = [](size_t bytes) { return (bytes + 511) & ~(size_t)255; };
  size_t total = 0;
  for (const auto &q : pieces) total += room(q.second);
  // new memory, which may come to lie at the old address (as after a run that did
  // not fit), holds no box table
  if (total > arena.cap) uploaded_sig.clear();
  arena.ensure(total);
  each_buf([](DevBuf &b) {
    if (b.view) b.release();
  });
  total = 0;
  for (const auto &q : pieces) {
    q.first->place(arena, total, room(q.second));
    total += room(q.second);
  }
}

// Host memory for `bytes` read back from the device: pinned once the plan's first
// run has ended, else `unpinned`.
unsigned char *Plan::host_room(size_t bytes, std::vector<unsigned char> &unpinned) {
  if (runs > 0) pinned.ensure(bytes);
  if (pinned.p && pinned.cap >= bytes) return static_cast<unsigned char *>(pinned.p);
  unpinned.resize(bytes);
  return unpinned.data();
}

void Plan::read_back(cudaStream_t s, bool timed) {
  const int nbox = (int)boxes_host.size();
  struct {
    Counters c;
    unsigned long long ngroups, nwarn;
  } hc;
  DevScal hs_;
  std::vector<unsigned char> unpinned;
  unsigned char *small = host_room(at_bucket, unpinned);
  CMH_CUDA(cudaMemcpyAsync(small, scal.p, at_bucket, cudaMemcpyDeviceToHost, s));
  CMH_CUDA(cudaStreamSynchronize(s));
  runs++;
  memcpy(&hs_, small, sizeof hs_);
  memcpy(&hc, small + at_ctr, sizeof hc);
  boxd_host.resize(7 * nbox);
  memcpy(boxd_host.data(), small + at_boxd, sizeof(uint32_t) * 7 * nbox);
  last = hs_;
  // CMH_FAULT=overflow: the run is treated as having outgrown its buffers, so
  // it is repeated with room until the attempts run out (CMH_ERR_CAPACITY),
  // as a rank whose receive buffer overflows stops (read_data.c:551-556)
  if (fault_active("overflow")) last.overflow |= 1u;
  if (hc.c.uf_giveups)
    fail(CMH_ERR_DEVICE_TIMEOUT, "union-find retry loop reached its iteration cap");
  if (hs_.failed)
    fail(CMH_ERR_DEVICE_TIMEOUT, hs_.next_tile == 0  // (the gather takes no tile then)
                                     ? "radix sort look-back wait reached its cap"
                                     : "run count look-back wait reached its cap");
  stats = cmh_stats{};
  stats.n_in = n_total;
  stats.n_out = n_total - hs_.kept_total;
  stats.n_images = hs_.img_total;
  stats.n_proc = hs_.np;
  stats.n_cells = hs_.R;
  stats.n_groups = (int64_t)hc.ngroups;
  stats.n_candidates = hs_.nc;
  stats.nhalos = hs_.nh;
  stats.n_edge_warn = (int64_t)hc.nwarn;
  stats.n_pair_tests = (int64_t)hc.c.pair_tests;
  stats.n_rechecks = (int64_t)hc.c.rechecks;
  stats.n_member_conflicts = (int64_t)hc.c.member_conflicts;
  stats.cell_factor = boxes_host[0].g.k;
  stats.key_bits = key_bits;
  stats.n_cell_pairs = (int64_t)hc.c.cand_pairs;
  stats.n_root_skips = (int64_t)hc.c.root_skips;
  stats.n_unions = (int64_t)hc.c.unions;
  stats.n_find_steps = (int64_t)hc.c.find_steps;
  stats.n_scan_iters = (int64_t)hc.c.scan_iters;
  stats.n_window_iters = (int64_t)hc.c.window_iters;
  stats.n_dense_tops = hs_.nd;
  stats.n_queued = (int64_t)hs_.qcount;
  stats.n_big_tops = hs_.nbig;
  if (timed) {
    float ms = 0;
    CMH_CUDA(cudaEventElapsedTime(&ms, ev0, ev1));
    stats.ms_total = ms;
    cudaEvent_t b[9] = {ev0, stage_ev[0], stage_ev[1], stage_ev[2], stage_ev[3],
                        stage_ev[4], stage_ev[5], stage_ev[6], ev1};
    for (int q = 0; q < 8; q++) CMH_CUDA(cudaEventElapsedTime(&stats.stage_ms[q], b[q], b[q + 1]));
  }
  out_nhalos = hs_.nh;
}

void Plan::run_batch(const std::vector<BoxSpec> &specs, int want_member, cudaStream_t s) {
  CMH_CUDA(cudaSetDevice(device));
  overwritten = false;
  struct Room {
    const Plan *plan;
    ~Room() { dense_room(plan, plan->device, 0); }
  } room{this};
  for (int attempt = 0; attempt < 3; attempt++) {
    prepare(specs, want_member);
    // the graph stays valid while the inputs, sizes and capacities do
    std::vector<unsigned char> sig(sizeof(BoxDev) * boxes_host.size());
    memcpy(sig.data(), boxes_host.data(), sig.size());
    int64_t samp_bits[3] = {0, 0, 0};
    memcpy(&samp_bits[0], &samp_in, 8);
    memcpy(&samp_bits[1], &samp_out, 8);
    samp_bits[2] = (int64_t)samp_seed ^ ((int64_t)samp_closed << 40);
    stall_sort = fault_active("lookback");
    stall_gather = fault_active("gather");
    const int64_t caps[12] = {np_cap, nd_cap, nc_cap, (int64_t)want_member, (int64_t)fp32,
                              (int64_t)dense_min, (int64_t)vel_wait,
                              sampling ? samp_bits[0] : -1, samp_bits[1],
                              samp_bits[2] ^ (int64_t)(uintptr_t)samp_ids,
                              (int64_t)spin_cap,
                              (int64_t)stall_sort | (int64_t)stall_gather << 1};
    sig.insert(sig.end(), (const unsigned char *)caps, (const unsigned char *)caps + sizeof caps);
    // and the workspace addresses the recorded launches use
    each_buf([&](DevBuf &b) {
      sig.insert(sig.end(), (const unsigned char *)&b.p, (const unsigned char *)&b.p + sizeof b.p);
    });
    sig.insert(sig.end(), (const unsigned char *)ltab_all.data(),
               (const unsigned char *)(ltab_all.data() + ltab_all.size()));
    int slot = -1;  // the recorded graph of this shape, if any
    for (int q = 0; q < 2; q++)
      if (graph_exec[q] && sig == graph_sig[q]) slot = q;
    const bool same = slot >= 0;
    // the device box table (and length tables) hold the last uploaded shape,
    // which an eager run of another shape may have replaced since the graph
    // was recorded: upload whenever they differ from this run's
    if (sig != uploaded_sig) {
      uploaded_sig.clear();
      CMH_CUDA(cudaMemcpyAsync(b_boxes.p, boxes_host.data(), sizeof(BoxDev) * boxes_host.size(),
                               cudaMemcpyHostToDevice, s));
      if (varlink)
        CMH_CUDA(cudaMemcpyAsync(ltab_dev.p, ltab_all.data(), ltab_all.size() * sizeof(double),
                                 cudaMemcpyHostToDevice, s));
      CMH_CUDA(cudaStreamSynchronize(s));
      uploaded_sig = sig;
    }
    const long long l0 = g_launches;
    if (use_graph && same) {
      // a replay is timed as a whole; stage times come from eager runs
      CMH_CUDA(cudaEventRecord(ev0, s));
      CMH_CUDA(cudaGraphLaunch(graph_exec[slot], s));
      graph_next = 1 - slot;  // keep the one just used
      CMH_CUDA(cudaEventRecord(ev1, s));
      launches_per_run_graph_ok = true;
      queue_pending();
      read_back(s, false);
      CMH_CUDA(cudaEventElapsedTime(&stats.ms_total, ev0, ev1));
    } else {
      if (pos_dtype == CMH_FLOAT64) issue<double>(want_member, s, true);
      else issue<float>(want_member, s, true);
      queue_pending();
      read_back(s, true);
      launches_per_run = (int32_t)(g_launches - l0);
      if (!(last.overflow & 1u) && use_graph) capture(want_member, s, sig);
    }
    stats.n_launches = launches_per_run;
    if (last.overflow & 2u)  // faster next time, within the rows budget
      nd_cap = std::min<int64_t>((int64_t)last.nd + last.nd / 4 + 256,
                                 std::max<int64_t>(nd_cap, rows_cap_for(np_cap, k3all)));
    if (!(last.overflow & 1u)) return;
    np_cap = (int64_t)last.np_raw + last.np_raw / 8 + 4096;  // repeat with room
    if (overwritten) {
      // one input buffer, already refilled with the next run's inputs: this
      // run's are copied again, and the next run's wait for the repeat
      CMH_CUDA(cudaStreamSynchronize(side_stream));
      staged.front().pending = true;
      overwritten = false;
      stage_inputs(cur_host.data(), (int)cur_host.size(), s, 0);
      CMH_CUDA(cudaStreamWaitEvent(s, ev_pos[0], 0));
      ev_vel_ready = ev_vel[0];
    }
  }
  fail(CMH_ERR_CAPACITY, "processed particles kept outgrowing the buffers");
}

void Plan::capture(int want_member, cudaStream_t s, const std::vector<unsigned char> &sig) {
  const int q = graph_next;
  graph_next = 1 - q;
  if (graph_exec[q]) {
    cudaGraphExecDestroy(graph_exec[q]);
    graph_exec[q] = nullptr;
    graph_sig[q].clear();
  }
  // recorded on the plan's own stream (the legacy stream cannot be
  // captured); the graph is then launched on the caller's stream
  if (!cap_stream) CMH_CUDA(cudaStreamCreateWithFlags(&cap_stream, cudaStreamNonBlocking));
  cudaGraph_t graph = nullptr;
  CMH_CUDA(cudaStreamBeginCapture(cap_stream, cudaStreamCaptureModeThreadLocal));
  try {
    if (pos_dtype == CMH_FLOAT64) issue<double>(want_member, cap_stream, false);
    else issue<float>(want_member, cap_stream, false);
  } catch (...) {
    cudaStreamEndCapture(cap_stream, &graph);
    if (graph) cudaGraphDestroy(graph);
    throw;
  }
  CMH_CUDA(cudaStreamEndCapture(cap_stream, &graph));
  cudaError_t e = cudaGraphInstantiate(&graph_exec[q], graph, 0);
  cudaGraphDestroy(graph);
  CMH_CUDA(e);
  graph_sig[q] = sig;
  (void)s;
}

// Grid search over the cell-size scale and the dense-top threshold, timing
// eager runs of the real boxes (after one untimed run per setting, which
// also grows the buffers).  The fastest setting stays in the plan.
cmh_tuning Plan::autotune(const std::vector<BoxSpec> &specs, int repeats, cudaStream_t s) {
  const double scales[] = {0.5, 0.75, 1.0, 1.5, 2.0};
  const uint32_t mins[] = {8, 16, 32};
  const bool graph0 = use_graph;
  use_graph = false;
  cmh_tuning best{cell_scale, (int32_t)dense_min, 1e30f, 0};
  for (double sc : scales)
    for (uint32_t dm : mins) {
      cell_scale = sc;
      dense_min = dm;
      // each setting starts from an empty workspace, so that one setting's
      // large buffers (many top cells, or many dense ones) do not stay allocated
      // under the next; a setting that does not fit in memory is skipped
      release_workspace();
      float t = 0;
      try {
        run_batch(specs, 0, s);
        for (int r = 0; r < std::max(repeats, 1); r++) {
          run_batch(specs, 0, s);
          t += stats.ms_total;
        }
      } catch (const Error &e) {
        if (e.code != CMH_ERR_OUT_OF_MEMORY) {
          use_graph = graph0;
          throw;
        }
        continue;
      }
      t /= std::max(repeats, 1);
      best.tried++;
      if (t < best.ms) {
        best.ms = t;
        best.cell_scale = sc;
        best.dense_min = (int32_t)dm;
      }
    }
  release_workspace();
  use_graph = graph0;
  if (best.tried == 0) fail(CMH_ERR_OUT_OF_MEMORY, "no setting of the autotuner fits in memory");
  cell_scale = best.cell_scale;
  dense_min = (uint32_t)best.dense_min;
  return best;
}

namespace {
// Byte offsets of each box's positions and velocities in the input buffers
// (256-byte aligned slices); returns the totals.
void input_layout(const cmh_particles *parts, int nbox, std::vector<size_t> *opos,
                  std::vector<size_t> *ovel, size_t *tpos, size_t *tvel) {
  size_t p = 0, v = 0;
  opos->resize(nbox);
  ovel->resize(nbox);
  for (int i = 0; i < nbox; i++) {
    (*opos)[i] = p;
    (*ovel)[i] = v;
    p += ((size_t)parts[i].n * 3 * (parts[i].pos_dtype == CMH_FLOAT64 ? 8 : 4) + 255) & ~(size_t)255;
    v += ((size_t)parts[i].n * 3 * (parts[i].vel_dtype == CMH_FLOAT64 ? 8 : 4) + 255) & ~(size_t)255;
  }
  *tpos = p;
  *tvel = v;
}

bool same_inputs(const std::vector<cmh_particles> &a, const cmh_particles *b, int nbox) {
  if ((int)a.size() != nbox) return false;
  for (int i = 0; i < nbox; i++)
    if (a[i].pos != b[i].pos || a[i].vel != b[i].vel || a[i].n != b[i].n ||
        a[i].pos_dtype != b[i].pos_dtype || a[i].vel_dtype != b[i].vel_dtype)
      return false;
  return true;
}
}  // namespace

void Plan::ensure_side() {
  if (side_stream) return;
  CMH_CUDA(cudaStreamCreateWithFlags(&side_stream, cudaStreamNonBlocking));
  CMH_CUDA(cudaEventCreateWithFlags(&ev_side_start, cudaEventDisableTiming));
  CMH_CUDA(cudaEventCreateWithFlags(&ev_pos_free, cudaEventDisableTiming));
  CMH_CUDA(cudaEventCreateWithFlags(&ev_vel_free, cudaEventDisableTiming));
  for (int b = 0; b < 2; b++) {
    CMH_CUDA(cudaEventCreateWithFlags(&ev_pos[b], cudaEventDisableTiming));
    CMH_CUDA(cudaEventCreateWithFlags(&ev_vel[b], cudaEventDisableTiming));
  }
}

int Plan::stage_inputs(const cmh_particles *parts, int nbox, cudaStream_t s, int b) {
  CMH_CUDA(cudaSetDevice(device));
  ensure_side();
  std::vector<size_t> opos, ovel;
  size_t tpos, tvel;
  input_layout(parts, nbox, &opos, &ovel, &tpos, &tvel);
  in_pos[b].ensure(std::max<size_t>(tpos, 256));
  in_vel[b].ensure(std::max<size_t>(tvel, 256));
  // after the caller's queued work (a run that read this buffer before), on
  // the side stream: the positions first, at the link's full bandwidth
  CMH_CUDA(cudaEventRecord(ev_side_start, s));
  CMH_CUDA(cudaStreamWaitEvent(side_stream, ev_side_start, 0));
  copy_inputs(parts, nbox, b, false);
  return b;
}

// The copies of staged host inputs into buffer b on the side stream, every
// box's positions before any velocities.  `behind_run`: the positions wait
// for the queued run's ingest and the velocities for its property sums.
void Plan::copy_inputs(const cmh_particles *parts, int nbox, int b, bool behind_run) {
  std::vector<size_t> opos, ovel;
  size_t tpos, tvel;
  input_layout(parts, nbox, &opos, &ovel, &tpos, &tvel);
  if (behind_run) CMH_CUDA(cudaStreamWaitEvent(side_stream, ev_pos_free, 0));
  for (int i = 0; i < nbox; i++)
    if (parts[i].n > 0)
      CMH_CUDA(cudaMemcpyAsync(in_pos[b].as<unsigned char>() + opos[i], parts[i].pos,
                               (size_t)parts[i].n * 3 * (parts[i].pos_dtype == CMH_FLOAT64 ? 8 : 4),
                               cudaMemcpyHostToDevice, side_stream));
  CMH_CUDA(cudaEventRecord(ev_pos[b], side_stream));
  if (behind_run) CMH_CUDA(cudaStreamWaitEvent(side_stream, ev_vel_free, 0));
  for (int i = 0; i < nbox; i++)
    if (parts[i].n > 0)
      CMH_CUDA(cudaMemcpyAsync(in_vel[b].as<unsigned char>() + ovel[i], parts[i].vel,
                               (size_t)parts[i].n * 3 * (parts[i].vel_dtype == CMH_FLOAT64 ? 8 : 4),
                               cudaMemcpyHostToDevice, side_stream));
  CMH_CUDA(cudaEventRecord(ev_vel[b], side_stream));
}

void Plan::queue_pending() {
  // (a run on device-resident particles records no free events: what is
  // staged waits for the next run on host inputs)
  if (input_buffers != 1 || !vel_wait || staged.empty() || !staged.front().pending) return;
  Staged &f = staged.front();
  std::vector<size_t> opos, ovel;
  size_t tpos, tvel;
  input_layout(f.parts.data(), (int)f.parts.size(), &opos, &ovel, &tpos, &tvel);
  // the buffer is in use by the queued run: it is not grown now (a larger
  // next run is copied when it starts)
  if (tpos > in_pos[0].cap || tvel > in_vel[0].cap) return;
  copy_inputs(f.parts.data(), (int)f.parts.size(), 0, true);
  f.pending = false;
  overwritten = true;
}

std::vector<cmh_particles> Plan::take_inputs(const cmh_particles *parts, int nbox,
                                             cudaStream_t s) {
  int b = -1;
  cur_host.assign(parts, parts + nbox);
  overwritten = false;
  if (!staged.empty()) {
    const Staged &f = staged.front();
    if (same_inputs(f.parts, parts, nbox)) {
      if (!f.pending) b = f.buf;  // else copied now, below
      staged.erase(staged.begin());
    } else {
      // not what was staged: the staged copies are dropped
      CMH_CUDA(cudaStreamSynchronize(side_stream));
      staged.clear();
    }
  }
  // not staged: copied now, into the first buffer (a plan that is never
  // given prefetches keeps a single input buffer)
  if (b < 0) b = stage_inputs(parts, nbox, s, 0);
  last_buf = b;
  CMH_CUDA(cudaStreamWaitEvent(s, ev_pos[b], 0));
  ev_vel_ready = ev_vel[b];
  vel_wait = true;
  std::vector<size_t> opos, ovel;
  size_t tpos, tvel;
  input_layout(parts, nbox, &opos, &ovel, &tpos, &tvel);
  std::vector<cmh_particles> dp(parts, parts + nbox);
  for (int i = 0; i < nbox; i++) {
    dp[i].pos = in_pos[b].as<unsigned char>() + opos[i];
    dp[i].vel = in_vel[b].as<unsigned char>() + ovel[i];
    dp[i].location = CMH_DEVICE;
  }
  return dp;
}

void Plan::run(const cmh_particles &parts, int want_member, cudaStream_t s) {
  BoxSpec sp;
  sp.params = params;
  sp.ltab = ltab_host;
  sp.pos = parts.pos;
  sp.vel = parts.vel;
  sp.vel_f64 = parts.vel_dtype == CMH_FLOAT64;
  sp.n = parts.n;
  sp.cell_factor = 0;
  run_batch({sp}, want_member, s);
}

}  // namespace cmh
