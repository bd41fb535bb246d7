// FoF group labels for small particle sets without any device allocation.
//
// Some callers cannot call cudaMalloc: a process whose framework has already
// reserved nearly all device memory for its own caching allocator, a service
// that forbids allocation after start-up so that latency stays flat, or a
// plugin host that only lends out buffers it owns.  For them this variant
// keeps its scratch -- union-find parents, cell lists and error flags -- in
// one file-scope device array of fixed size that every GPU loading the
// library holds until the process exits.  The caller still passes the input
// positions and the output label array (device memory it owns).
//
// Limits: at most kMaxParticles particles and a cell grid of at most
// kMaxCells cells (the cell side grows to fit).  Non-periodic only.
//
// Method.  Particles are put into fine cells of side h <= l / sqrt(3), as in
// the main path: two particles of a fine cell are linked wherever they sit in
// it.  The occupied fine cells are found through a hash table whose slots
// hold the lowest particle of a cell (the cell's coordinates are recomputed
// from that particle's position, so no keys are kept), and the union-find runs
// over those lowest particles.  Each cell looks its 62 forward neighbours
// up, the 13 at distance 1 before the other 49, and pairs of cells in
// different components are tested as in the main path: 32 at a time, by one
// lane each for a bounded number of steps, then by the whole warp.  The
// coarse cells of the grid above hold thousands of particles where a clump
// sits, and walking their lists for every particle pair took 16 to 46 ms for
// 50,021 particles of the benchmark's distribution, where a call now takes
// 0.14 ms (eight kernels of 3 to 42 us).
//
// Sharing: every call on a device uses the same array.  Each call clears what
// must start empty before use, but two calls whose work overlaps on the GPU
// (for instance on two streams) race on the array and give wrong labels.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <mutex>

#include "cmh_internal.cuh"
#include "fof_kernels.cuh"

namespace cmh {
namespace {

constexpr int kMaxParticles = 1 << 16;
constexpr int kMaxCells = 1 << 18;
constexpr int kThreads = 256;

constexpr int kTableBits = 17;
constexpr uint32_t kSlots = 1u << kTableBits;  // twice the particles: probes stay short
constexpr uint32_t kNone = 0xffffffffu;

struct NoAllocScratch {
  uint32_t parent[kMaxParticles];
  uint32_t next[kMaxParticles];
  union {
    uint32_t cell_head[kMaxCells];  // grid path
    struct {                        // fine-cell path
      uint32_t table[kSlots];          // lowest particle of the slot's fine cell
      uint32_t order[kMaxParticles];   // particles cell by cell
      uint32_t span[kMaxParticles];    // at a cell's lowest particle: its particles' count,
                                       // then (first in order) << 16 | (count - 1)
    };
  };
  uint32_t cells;       // fine-cell path: entries of `order` given out
  // what the host reads back
  Counters ctr;         // uf_giveups is the error flag of the union loop
  unsigned int flags[4];  // [0] particles outside the padded domain
};

static __device__ __align__(256) NoAllocScratch g_noalloc;

// Host-side address of g_noalloc on each device, looked up with that device
// current.  In host code the symbol itself is only a stand-in, never a device
// address.  The lookup is redone only when the device's context changed (a
// cudaDeviceReset followed by new work loads the module again, and the array
// may then sit elsewhere); the context is told apart by its ID, which the
// driver never reuses within a process.
std::mutex g_addr_mutex;
struct ScratchAddr {
  NoAllocScratch *p = nullptr;
  unsigned long long ctx_id = 0;
};
ScratchAddr g_addr[128];

// ID of the calling thread's current context, 0 when none is current.
unsigned long long current_context_id() {
  typedef CUresult(CUDAAPI * CtxGetCurrent)(CUcontext *);
  typedef CUresult(CUDAAPI * CtxGetId)(CUcontext, unsigned long long *);
  static CtxGetCurrent get_current = nullptr;
  static CtxGetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", (void **)&get_current, cudaEnableDefault,
                                &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      get_current = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", (void **)&get_id, cudaEnableDefault, &q) !=
            cudaSuccess || q != cudaDriverEntryPointSuccess)
      get_id = nullptr;
  });
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
  if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

NoAllocScratch *scratch_on(int device) {
  std::lock_guard<std::mutex> lock(g_addr_mutex);
  if (device < 0 || device >= 128) fail(CMH_ERR_INVALID_ARGUMENT, "device index out of range");
  ScratchAddr &a = g_addr[device];
  const unsigned long long id = current_context_id();
  if (!a.p || id == 0 || id != a.ctx_id) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc);
    if (e != cudaSuccess || !p)
      fail(CMH_ERR_CUDA, std::string("cudaGetSymbolAddress of the scratch array failed: ") +
                             cudaGetErrorString(e));
    a.p = static_cast<NoAllocScratch *>(p);
    a.ctx_id = current_context_id();  // the lookup made the primary context current
  }
  return a.p;
}

struct NaGrid {
  double rmin[3], lc;
  int nc[3];
  double rmax[3];
  double linksq;
};

__global__ void k_na_clear(NoAllocScratch *sc, int n, int ncell) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ncell; i += stride)
    sc->cell_head[i] = 0xffffffffu;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    sc->parent[i] = (uint32_t)i;
    sc->next[i] = 0xffffffffu;
  }
  if (blockIdx.x == 0 && threadIdx.x < 4) sc->flags[threadIdx.x] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->ctr = Counters{};
}

template <class PT>
__device__ __forceinline__ int na_cell(const NaGrid &g, const PT *pos, int i, int c[3]) {
  for (int a = 0; a < 3; a++) {
    const double x = (double)pos[3 * i + a];
    if (!(x >= g.rmin[a] && x <= g.rmax[a])) return -1;
    int k = (int)floor(__ddiv_rn(__dsub_rn(x, g.rmin[a]), g.lc));
    c[a] = k < 0 ? 0 : (k >= g.nc[a] ? g.nc[a] - 1 : k);
  }
  return (c[2] * g.nc[1] + c[1]) * g.nc[0] + c[0];
}

template <class PT>
__global__ void k_na_bin(NoAllocScratch *sc, const PT *pos, int n, NaGrid g) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int c[3];
    const int cell = na_cell(g, pos, i, c);
    if (cell < 0) {
      atomicAdd(&sc->flags[0], 1u);
      continue;
    }
    sc->next[i] = atomicExch(&sc->cell_head[cell], (uint32_t)i);
  }
}

// The reference's pair predicate in double (FOF.c:351-357), dx in the
// storage precision.
template <class PT>
__device__ __forceinline__ bool na_linked(const PT *pos, int i, int j, double linksq) {
  double d[3];
  for (int a = 0; a < 3; a++) {
    if constexpr (sizeof(PT) == 4) d[a] = (double)__fsub_rn(pos[3 * i + a], pos[3 * j + a]);
    else d[a] = __dsub_rn(pos[3 * i + a], pos[3 * j + a]);
  }
  const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])),
                              __dmul_rn(d[2], d[2]));
  return !(d2 > linksq);
}

template <class PT>
__global__ void k_na_befriend(NoAllocScratch *sc, const PT *pos, int n, NaGrid g) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int c[3];
    if (na_cell(g, pos, i, c) < 0) continue;
    for (int dz = -1; dz <= 1; dz++)
      for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++) {
          const int x = c[0] + dx, y = c[1] + dy, z = c[2] + dz;
          if (x < 0 || y < 0 || z < 0 || x >= g.nc[0] || y >= g.nc[1] || z >= g.nc[2]) continue;
          for (uint32_t j = sc->cell_head[(z * g.nc[1] + y) * g.nc[0] + x]; j != 0xffffffffu;
               j = sc->next[j]) {
            if ((int)j <= i) continue;  // each unordered pair once
            if (uf_find(sc->parent, (uint32_t)i) == uf_find(sc->parent, j)) continue;
            if (na_linked(pos, i, (int)j, g.linksq)) uf_union(sc->parent, (uint32_t)i, j, &sc->ctr);
          }
        }
  }
}

// label = root = lowest index of the group (hook-to-min union-find)
__global__ void k_na_label(NoAllocScratch *sc, int n, uint32_t *label) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    label[i] = uf_find(sc->parent, (uint32_t)i);
}

// ---- fine-cell path ----

struct FineGrid {
  double rmin[3], rmax[3];
  double h, inv_h;
  double linksq, prune_sq;  // prune_sq: as Geom's
};

struct FineCell {
  long long c[3];
};
__device__ __forceinline__ bool operator==(const FineCell &a, const FineCell &b) {
  return a.c[0] == b.c[0] && a.c[1] == b.c[1] && a.c[2] == b.c[2];
}

template <class PT>
__device__ __forceinline__ FineCell na_fine(const FineGrid &g, const PT *pos, uint32_t i) {
  FineCell f;
#pragma unroll
  for (int a = 0; a < 3; a++)
    f.c[a] = (long long)floor(__dmul_rn(__dsub_rn((double)pos[3 * i + a], g.rmin[a]), g.inv_h));
  return f;
}

// Multiplicative hash of a cell's coordinates (the high bits of the product are
// the best mixed).  The odd constants are published ones: 2^64 over the golden
// ratio (Fibonacci hashing, Knuth, The Art of Computer Programming 3, 6.4) and two
// of the 64-bit primes of xxHash (Collet).
__device__ __forceinline__ uint32_t na_hash(const FineCell &f) {
  uint64_t x = (uint64_t)f.c[0] * 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 32)) + (uint64_t)f.c[1] * 0xC2B2AE3D27D4EB4Full;
  x = (x ^ (x >> 29)) + (uint64_t)f.c[2] * 0x165667B19E3779F9ull;
  x *= 0x9E3779B97F4A7C15ull;
  return (uint32_t)(x >> (64 - kTableBits));
}

__global__ void k_na_fine_clear(NoAllocScratch *sc, int n) {
  const int stride = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
  uint4 *tab = reinterpret_cast<uint4 *>(sc->table);
  for (int i = t; i < (int)kSlots / 4; i += stride) tab[i] = make_uint4(kNone, kNone, kNone, kNone);
  for (int i = t; i < n; i += stride) sc->span[i] = 0u;
  if (t < 4) sc->flags[t] = 0;
  if (t == 0) {
    sc->cells = 0;
    sc->ctr = Counters{};
  }
}

// Puts every particle into the hash table; next[i] becomes its slot.  Particles
// number at most half the slots, so every probe ends.
template <class PT>
__global__ void __launch_bounds__(kThreads) k_na_fine_insert(NoAllocScratch *sc, const PT *pos,
                                                             int n, FineGrid g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool in = true;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double x = (double)pos[3 * i + a];
    in &= x >= g.rmin[a] && x <= g.rmax[a];  // NaN is outside
  }
  if (!in) {
    atomicAdd(&sc->flags[0], 1u);
    sc->next[i] = kNone;
    return;
  }
  const FineCell f = na_fine(g, pos, (uint32_t)i);
  uint32_t s = na_hash(f);
  for (uint32_t probe = 0; probe < kSlots; probe++, s = (s + 1) & (kSlots - 1)) {
    uint32_t v = __ldcg(sc->table + s);
    if (v == kNone) v = atomicCAS(sc->table + s, kNone, (uint32_t)i);
    if (v == kNone) break;
    // whichever particle the slot holds, it is one of the slot's cell
    if (na_fine(g, pos, v) == f) {
      if (v > (uint32_t)i) atomicMin(sc->table + s, (uint32_t)i);
      break;
    }
  }
  sc->next[i] = s;
}

// Particles per cell, each particle's rank in its cell (kept in parent) and
// its cell's lowest particle (in next).
__global__ void __launch_bounds__(kThreads) k_na_fine_count(NoAllocScratch *sc, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = sc->next[i];
  if (s == kNone) return;
  const uint32_t lo = sc->table[s];
  sc->next[i] = lo;
  sc->parent[i] = atomicAdd(sc->span + lo, 1u);
}

// A place in `order` for every cell (the cells' order does not matter): one
// atomic per warp.
__global__ void __launch_bounds__(kThreads) k_na_fine_place(NoAllocScratch *sc, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const uint32_t cnt = i < n && sc->next[i] == (uint32_t)i ? sc->span[i] : 0u;
  uint32_t inc = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  uint32_t base = 0;
  if (lane == 31 && inc) base = atomicAdd(&sc->cells, inc);
  base = __shfl_sync(0xffffffffu, base, 31);
  if (cnt) sc->span[i] = (base + inc - cnt) << 16 | (cnt - 1u);
}

// Particles into their places; the union-find starts with every cell alone.
__global__ void __launch_bounds__(kThreads) k_na_fine_fill(NoAllocScratch *sc, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t lo = sc->next[i];
  if (lo != kNone) sc->order[(sc->span[lo] >> 16) + sc->parent[i]] = (uint32_t)i;
  sc->parent[i] = lo == kNone ? (uint32_t)i : lo;
}

// The lowest particle of fine cell f, kNone when it is empty.
template <class PT>
__device__ __forceinline__ uint32_t na_lookup(const NoAllocScratch *sc, const FineGrid &g,
                                              const PT *pos, const FineCell &f) {
  uint32_t s = na_hash(f);
  for (uint32_t probe = 0; probe < kSlots; probe++, s = (s + 1) & (kSlots - 1)) {
    const uint32_t v = sc->table[s];
    if (v == kNone) return kNone;
    if (na_fine(g, pos, v) == f) return v;
  }
  return kNone;
}

// Whether a particle may be linked to one of fine cell f (its distance from
// the cell's box against the linking length).
template <class PT>
__device__ __forceinline__ bool na_near(const FineGrid &g, const PT *pos, uint32_t i,
                                        const FineCell &f) {
  double q = 0.0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double x = (double)pos[3 * i + a], lo = g.rmin[a] + (double)f.c[a] * g.h;
    const double e = fmax(0.0, fmax(lo - x, x - (lo + g.h)));
    q += e * e;
  }
  return !(q > g.prune_sq);
}

constexpr int kSoloSteps = 48;  // steps of one lane on a cell pair before the warp takes it

// Tests the listed cell pairs, n <= 32, and joins the linked ones.
template <class PT>
__device__ __forceinline__ void na_drain(NoAllocScratch *sc, const FineGrid &g, const PT *pos,
                                         const uint2 *pairs, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t a = 0, b = 0, sa = 0, sb = 0;
  bool open = false;
  if (lane < n) {
    a = pairs[lane].x;
    b = pairs[lane].y;
    sa = sc->span[a];
    sb = sc->span[b];
    if ((sb & 0xffffu) < (sa & 0xffffu)) {  // a: the cell with fewer particles
      uint32_t t = a;
      a = b;
      b = t;
      t = sa;
      sa = sb;
      sb = t;
    }
    if (uf_find(sc->parent, a) != uf_find(sc->parent, b)) {
      const FineCell fb = na_fine(g, pos, b);
      int left = kSoloSteps;
      bool hit = false;
      for (uint32_t p = 0; p <= (sa & 0xffffu) && !hit && left > 0; p++, left--) {
        const uint32_t i = sc->order[(sa >> 16) + p];
        if (!na_near(g, pos, i, fb)) continue;
        for (uint32_t q = 0; q <= (sb & 0xffffu) && !hit && left > 0; q++, left--)
          hit = na_linked(pos, (int)i, (int)sc->order[(sb >> 16) + q], g.linksq);
      }
      if (hit) uf_union(sc->parent, a, b, &sc->ctr);
      else open = left <= 0;
    }
  }
  for (uint32_t todo = __ballot_sync(0xffffffffu, open); todo; todo &= todo - 1u) {
    const int l = __ffs(todo) - 1;
    const uint32_t la = __shfl_sync(0xffffffffu, a, l), lb = __shfl_sync(0xffffffffu, b, l);
    const uint32_t lsa = __shfl_sync(0xffffffffu, sa, l), lsb = __shfl_sync(0xffffffffu, sb, l);
    if (__any_sync(0xffffffffu, uf_find(sc->parent, la) == uf_find(sc->parent, lb))) continue;
    const FineCell fb = na_fine(g, pos, lb);
    bool hit = false;
    for (uint32_t p0 = 0; p0 <= (lsa & 0xffffu) && !hit; p0 += 32) {
      const bool has = p0 + lane <= (lsa & 0xffffu);
      const uint32_t mine = has ? sc->order[(lsa >> 16) + p0 + lane] : 0u;
      for (uint32_t near = __ballot_sync(0xffffffffu, has && na_near(g, pos, mine, fb));
           near && !hit; near &= near - 1u) {
        const uint32_t i = __shfl_sync(0xffffffffu, mine, __ffs(near) - 1);
        for (uint32_t q0 = 0; q0 <= (lsb & 0xffffu) && !hit; q0 += 32) {
          const bool in = q0 + lane <= (lsb & 0xffffu);
          hit = __any_sync(0xffffffffu,
                           in && na_linked(pos, (int)i, (int)sc->order[(lsb >> 16) + q0 + lane],
                                           g.linksq));
        }
      }
    }
    if (hit && (int)lane == l) uf_union(sc->parent, la, lb, &sc->ctr);
    __syncwarp();
  }
}

// A warp takes the fine cells whose lowest particles are among kGroup consecutive
// particles, and their (cell, forward offset) pairs one per lane.  FAR false:
// the 13 offsets at distance 1; true: the 49 at distance 2.  The lookups are
// chains of dependent reads, so short groups (more warps) pay: both kernels
// together take 171 us for 50,021 particles with groups of 32, 87 of 8, 75
// of 4, 78 of 2.
constexpr int kGroup = 4;
template <class PT, bool FAR>
__global__ void __launch_bounds__(kThreads) k_na_fine_join(NoAllocScratch *sc, const PT *pos,
                                                           int n, FineGrid g) {
  constexpr uint32_t kOffsets = FAR ? 49 : 13;
  __shared__ uint2 s_pairs[kThreads / 32][64];
  __shared__ FineCell s_cell[kThreads / 32][kGroup];
  __shared__ uint32_t s_low[kThreads / 32][kGroup];
  // forward offsets (dz, dy, dx) in steps of the window 5 x 5 x 5, from its centre
  __shared__ uint8_t s_off[49];
  if (threadIdx.x == 0) {
    int m = 0;
    for (int o = 63; o < 125; o++) {
      const int dx = o % 5 - 2, dy = o / 5 % 5 - 2, dz = o / 25 - 2;
      const bool far = dx * dx > 1 || dy * dy > 1 || dz * dz > 1;
      if (far == FAR) s_off[m++] = (uint8_t)o;
    }
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, below = (1u << lane) - 1u;
  uint32_t npair = 0;
  const int warps = (int)(gridDim.x * (blockDim.x / 32));
  for (int i0 = (int)(blockIdx.x * (blockDim.x / 32) + w) * kGroup; i0 < n; i0 += warps * kGroup) {
    const int i = i0 + (int)lane;
    const bool low = (int)lane < kGroup && i < n && sc->next[i] == (uint32_t)i;
    const uint32_t lows = __ballot_sync(0xffffffffu, low);
    if (low) {
      const int at = __popc(lows & below);
      s_cell[w][at] = na_fine(g, pos, (uint32_t)i);
      s_low[w][at] = (uint32_t)i;
    }
    __syncwarp();
    const uint32_t items = (uint32_t)__popc(lows) * kOffsets;
    for (uint32_t j0 = 0; j0 < items; j0 += 32) {
      const uint32_t j = j0 + lane;
      bool apart = false;
      uint32_t a = 0, b = kNone;
      if (j < items) {
        a = s_low[w][j / kOffsets];
        FineCell f = s_cell[w][j / kOffsets];
        const int o = s_off[j % kOffsets];
        f.c[0] += o % 5 - 2;
        f.c[1] += o / 5 % 5 - 2;
        f.c[2] += o / 25 - 2;
        b = na_lookup(sc, g, pos, f);
        if (b != kNone) apart = uf_find(sc->parent, a) != uf_find(sc->parent, b);
      }
      const uint32_t m = __ballot_sync(0xffffffffu, apart);
      if (apart) s_pairs[w][npair + __popc(m & below)] = make_uint2(a, b);
      npair += __popc(m);
      if (npair >= 32) {
        __syncwarp();
        npair -= 32;
        na_drain(sc, g, pos, s_pairs[w] + npair, 32);
        __syncwarp();
      }
    }
    __syncwarp();
  }
  if (npair) na_drain(sc, g, pos, s_pairs[w], npair);
}

template <class PT>
void fine_labels(NoAllocScratch *sc, const PT *pos, int n, const FineGrid &g, uint32_t *label,
                 cudaStream_t s) {
  const unsigned grid = (unsigned)((n + kThreads - 1) / kThreads);
  k_na_fine_clear<<<grid_for(kSlots / 4, kThreads, 4), kThreads, 0, s>>>(sc, n);
  CMH_LAUNCHED();
  k_na_fine_insert<PT><<<grid, kThreads, 0, s>>>(sc, pos, n, g);
  CMH_LAUNCHED();
  k_na_fine_count<<<grid, kThreads, 0, s>>>(sc, n);
  CMH_LAUNCHED();
  k_na_fine_place<<<grid, kThreads, 0, s>>>(sc, n);
  CMH_LAUNCHED();
  k_na_fine_fill<<<grid, kThreads, 0, s>>>(sc, n);
  CMH_LAUNCHED();
  constexpr int per_cta = kThreads / 32 * kGroup;
  const unsigned gj = (unsigned)((n + per_cta - 1) / per_cta);
  k_na_fine_join<PT, false><<<gj, kThreads, 0, s>>>(sc, pos, n, g);
  CMH_LAUNCHED();
  k_na_fine_join<PT, true><<<gj, kThreads, 0, s>>>(sc, pos, n, g);
  CMH_LAUNCHED();
  k_na_label<<<grid, kThreads, 0, s>>>(sc, n, label);
  CMH_LAUNCHED();
}

}  // namespace
}  // namespace cmh

extern "C" cmh_status cmh_fof_labels_noalloc(const cmh_fof_params *params, const void *pos,
                                             int32_t pos_dtype, int64_t n, uint32_t *label,
                                             void *stream) {
  using namespace cmh;
  try {
    if (!params || (n > 0 && (!pos || !label)) || n < 0)
      fail(CMH_ERR_INVALID_ARGUMENT, "params, device positions and labels are required");
    if (pos_dtype != CMH_FLOAT32 && pos_dtype != CMH_FLOAT64)
      fail(CMH_ERR_INVALID_ARGUMENT, "unknown position dtype");
    if (params->periodic || params->varlink)
      fail(CMH_ERR_INVALID_ARGUMENT, "the allocation-free variant is non-periodic, constant l");
    if (!(params->linklength > 0) || !(params->boundary >= 0))
      fail(CMH_ERR_INVALID_ARGUMENT, "Linklength must be > 0 and Boundarysize >= 0");
    if (n > kMaxParticles)
      fail(CMH_ERR_CAPACITY, "the allocation-free variant takes at most 65536 particles");
    if (n == 0) return CMH_OK;
    int dev = 0;
    CMH_CUDA(cudaGetDevice(&dev));
    NoAllocScratch *sc = scratch_on(dev);
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    NaGrid g{};
    double ext[3];
    for (int a = 0; a < 3; a++) {
      g.rmin[a] = params->lo[a] - params->boundary;
      g.rmax[a] = params->hi[a] + params->boundary;
      ext[a] = g.rmax[a] - g.rmin[a];
      if (!(ext[a] > 0) || !std::isfinite(ext[a]))
        fail(CMH_ERR_INVALID_ARGUMENT, "empty or unbounded domain");
    }
    g.linksq = params->linklength * params->linklength;
    // Cells no smaller than the linking length (so the 27-cell scan sees
    // every linked pair), and at least as large as the side that spreads the
    // padded domain over kMaxCells cells.  Counts are formed in double and
    // checked before any conversion to int.
    g.lc = std::max(params->linklength, std::cbrt(ext[0] * ext[1] * ext[2] / (double)kMaxCells));
    double cells[3] = {0, 0, 0};
    for (int it = 0;; it++) {
      double total = 1.0;
      for (int a = 0; a < 3; a++) {
        cells[a] = std::floor(ext[a] / g.lc) + 1.0;
        total *= cells[a];
      }
      if (total <= (double)kMaxCells) break;
      if (it >= 64 || !std::isfinite(g.lc))
        fail(CMH_ERR_INVALID_ARGUMENT, "no cell grid of at most 2^18 cells covers the domain");
      g.lc *= 1.25;
    }
    for (int a = 0; a < 3; a++) g.nc[a] = (int)cells[a];  // each <= kMaxCells
    int64_t ncell = (int64_t)g.nc[0] * g.nc[1] * g.nc[2];
    const int ni = (int)n;
    // Fine cells: particles of one cell are within l of each other also when
    // their indices were rounded (an index q is off by at most 2^-51 q), and
    // none is linked beyond two cells away.  Domains of more than 2^40 fine
    // cells an axis, where that rounding would eat the margin, keep the grid.
    const double emax = std::max(ext[0], std::max(ext[1], ext[2]));
    const double h0 = params->linklength / std::sqrt(3.0), qmax = emax / h0;
    if (qmax < 0x1p40) {
      FineGrid fg{};
      for (int a = 0; a < 3; a++) {
        fg.rmin[a] = g.rmin[a];
        fg.rmax[a] = g.rmax[a];
      }
      fg.h = h0 * (1.0 - 0x1p-20 - qmax * 0x1p-49);
      fg.inv_h = 1.0 / fg.h;
      fg.linksq = g.linksq;
      const double reach = params->linklength * (1.0 + 1e-5 + qmax * 0x1p-49);
      fg.prune_sq = reach * reach;
      if (pos_dtype == CMH_FLOAT32) fine_labels(sc, (const float *)pos, ni, fg, label, s);
      else fine_labels(sc, (const double *)pos, ni, fg, label, s);
    } else {
      const unsigned grid = grid_for(ncell > n ? ncell : n, kThreads, 4);
      k_na_clear<<<grid, kThreads, 0, s>>>(sc, ni, (int)ncell);
      CMH_LAUNCHED();
      const unsigned gp = grid_for(n, kThreads, 4);
      if (pos_dtype == CMH_FLOAT32) {
        k_na_bin<float><<<gp, kThreads, 0, s>>>(sc, (const float *)pos, ni, g);
        CMH_LAUNCHED();
        k_na_befriend<float><<<gp, kThreads, 0, s>>>(sc, (const float *)pos, ni, g);
        CMH_LAUNCHED();
      } else {
        k_na_bin<double><<<gp, kThreads, 0, s>>>(sc, (const double *)pos, ni, g);
        CMH_LAUNCHED();
        k_na_befriend<double><<<gp, kThreads, 0, s>>>(sc, (const double *)pos, ni, g);
        CMH_LAUNCHED();
      }
      k_na_label<<<gp, kThreads, 0, s>>>(sc, ni, label);
      CMH_LAUNCHED();
    }
    struct {
      Counters ctr;
      unsigned int flags[4];
    } back{};
    static_assert(offsetof(NoAllocScratch, flags) - offsetof(NoAllocScratch, ctr) ==
                      sizeof(Counters), "the counters and the flags are read in one copy");
    CMH_CUDA(cudaMemcpyAsync(&back, &sc->ctr, sizeof back, cudaMemcpyDeviceToHost, s));
    CMH_CUDA(cudaStreamSynchronize(s));
    const unsigned int *flags = back.flags;
    const Counters &ctr = back.ctr;
    if (flags[0]) fail(CMH_ERR_DOMAIN, "particles outside [lo - Boundarysize, hi + Boundarysize]");
    if (ctr.uf_giveups) fail(CMH_ERR_DEVICE_TIMEOUT, "union-find retry loop reached its cap");
    return CMH_OK;
  } catch (const Error &e) {
    set_error(e.msg);
    return e.code;
  }
}
