// GPU voxelizer and packed-geometry validation (compiled with -fmad=false so every
// binary64 edge function and hit depth rounds exactly as the reference computes it).
//
// Follows src/geometry/voxelize.ts:1-199 and src/geometry/wall-links.ts:1-131:
//   per projection (u, v, axis) in {(x,y,z), (y,z,x), (z,x,y)}: rasterize every
//   triangle onto integer (u, v) columns with the half-open edge rule, collect the
//   hit depths per column, sort them, fill [ceil(h0), ceil(h1)) spans into a vote;
//   a cell is the mesh's kind when two of three projections agree and it is still
//   fluid (body before supports); then EQ x faces, FLOOR/EQ z faces, counts,
//   pull-direction wall masks, q offsets (halfway fractions) and the ascending
//   list of fluid cells next to the body.
// GPU shape: a warp shares the pixels of 32 triangles' boxes in the counting and
// filling passes, one thread per column for sort-and-fill, one thread per cell
// for the rest; prefix sums give CSR column offsets, q offsets and the boundary
// list in cell order.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <vector>

#include "pw_internal.h"
#include "pw_launch.h"

namespace pwhost {

static thread_local std::string g_error;

void set_error(const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_error = buf;
}

const char *last_error() { return g_error.c_str(); }

int cuda_status(cudaError_t e, const char *what) {
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    set_error("device allocation failed (%s)", what);
    return PW_ERR_OOM;
  }
  set_error("CUDA error %s in %s", cudaGetErrorString(e), what);
  return PW_ERR_CUDA;
}

// Temporaries of one voxelization come from the stream-ordered pool: freeing
// one never waits for the whole device, and the pool keeps up to 256 MB mapped
// between calls.
static cudaError_t tmp_alloc(void *p, size_t bytes, cudaStream_t s) {
  prepare_pool();
  return cudaMallocAsync(reinterpret_cast<void **>(p), bytes, s);
}

// The pool takes its place in the address space here, on a stream of its own.
void prepare_pool() {
  static std::mutex lock;
  static bool done[64];
  int dev = 0;
  std::lock_guard<std::mutex> hold(lock);
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || done[dev]) { cudaGetLastError(); return; }
  done[dev] = true;
  cudaMemPool_t pool;
  cudaStream_t s;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    uint64_t keep = 256ull << 20;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess) {
    void *p = nullptr;
    if (cudaMallocAsync(&p, 1024, s) == cudaSuccess) cudaFreeAsync(p, s);
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
  }
  cudaGetLastError();
}
static void tmp_free(void *p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

uint32_t multiprocessors() {
  static std::atomic<int> counts[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); dev = 0; }
  int n = counts[dev].load(std::memory_order_relaxed);
  if (!n) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 1;
    }
    counts[dev].store(n, std::memory_order_relaxed);
  }
  return (uint32_t)n;
}

Grid::~Grid() {
  cudaFree(cell_arrays);
  cudaFree(link_arrays);
}

// ------------------------------------------------------------------ pinned slots
namespace {
constexpr size_t kSlabSlots = 64;
// A slab's head, in its own first slot: no container to grow, so nothing here throws
// through a C entry.
struct PinnedSlab {
  PinnedSlab *next;
  uint64_t used;  // a bit a slot; bit 0, the head's own, is always set
  bool empty() const { return used == 1u; }
  char *slot(int k) { return reinterpret_cast<char *>(this) + (size_t)k * kPinnedSlot; }
};
static_assert(sizeof(PinnedSlab) <= kPinnedSlot, "the head fits a slot");
std::mutex g_pinned_lock;
PinnedSlab *g_pinned = nullptr;
}  // namespace

void *pinned_acquire() {
  std::lock_guard<std::mutex> hold(g_pinned_lock);
  PinnedSlab *slab = g_pinned;
  while (slab && !~slab->used) slab = slab->next;
  if (!slab) {
    void *p = nullptr;
    if (cudaHostAlloc(&p, kSlabSlots * kPinnedSlot, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    slab = static_cast<PinnedSlab *>(p);
    *slab = PinnedSlab{g_pinned, 1u};
    g_pinned = slab;
  }
  const int k = __builtin_ctzll(~slab->used);
  slab->used |= 1ull << k;
  std::memset(slab->slot(k), 0, kPinnedSlot);
  return slab->slot(k);
}

void pinned_release(void *slot) {
  std::lock_guard<std::mutex> hold(g_pinned_lock);
  bool other_empty = false;
  PinnedSlab **own = nullptr;
  for (PinnedSlab **at = &g_pinned; *at; at = &(*at)->next) {
    const ptrdiff_t off = static_cast<char *>(slot) - (*at)->slot(0);
    if (off > 0 && off < (ptrdiff_t)(kSlabSlots * kPinnedSlot)) {
      (*at)->used &= ~(1ull << (off / (ptrdiff_t)kPinnedSlot));
      own = at;
    } else if ((*at)->empty()) {
      other_empty = true;
    }
  }
  if (own && (*own)->empty() && other_empty) {
    PinnedSlab *gone = *own;
    *own = gone->next;
    cudaFreeHost(gone);
  }
}

// ------------------------------------------------------------------ scan
// Exclusive prefix sum of n uint32 values into out[0..n], out[n] the total, in
// three launches and without a host synchronisation: 4096-value block sums, one
// block over the sums, then each block's own scan from its offset.
constexpr int kScanThreads = 1024, kScanItems = 4;

__device__ __forceinline__ uint32_t warp_scan(uint32_t v) {  // inclusive
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= (uint32_t)o) v += t;
  }
  return v;
}

// Exclusive scan over a block of up to 1024 threads (whole warps); *total gets the sum.
// `warps` holds 33 words of shared memory, free again at the caller's next barrier.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *warps, uint32_t *total) {
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, nw = (blockDim.x + 31u) >> 5;
  const uint32_t inc = warp_scan(v);
  if (lane == 31u) warps[w] = inc;
  __syncthreads();
  if (w == 0u) {
    const uint32_t s = lane < nw ? warps[lane] : 0u;
    const uint32_t t = warp_scan(s);
    if (lane < nw) warps[lane] = t - s;
    if (lane == 31u) warps[32] = t;
  }
  __syncthreads();
  *total = warps[32];
  return warps[w] + inc - v;
}

__global__ void __launch_bounds__(kScanThreads) scan_sums(const uint32_t *in, uint32_t *sums, size_t n) {
  __shared__ uint32_t warps[33];
  const size_t base = (size_t)blockIdx.x * (kScanThreads * kScanItems) + threadIdx.x * kScanItems;
  uint32_t local = 0, total;
  for (int k = 0; k < kScanItems; k++) local += base + k < n ? in[base + k] : 0u;
  block_scan(local, warps, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// One block an array of block sums (array b at sums + b * blocks): its exclusive scan in
// place; its total to total_a[b] and total_b[b].
__global__ void __launch_bounds__(kScanThreads) scan_offsets(uint32_t *sums, uint32_t blocks, uint32_t *total_a,
                                                            uint32_t *total_b) {
  __shared__ uint32_t warps[33];
  uint32_t carry = 0;
  sums += (size_t)blockIdx.x * blocks;
  for (uint32_t base = 0; base < blocks; base += kScanThreads) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < blocks ? sums[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_scan(v, warps, &total);
    if (i < blocks) sums[i] = carry + ex;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    total_a[blockIdx.x] = carry;
    if (total_b) total_b[blockIdx.x] = carry;
  }
}

__global__ void __launch_bounds__(kScanThreads) scan_write(const uint32_t *in, uint32_t *out, const uint32_t *offsets,
                                                          size_t n) {
  __shared__ uint32_t warps[33];
  const size_t base = (size_t)blockIdx.x * (kScanThreads * kScanItems) + threadIdx.x * kScanItems;
  uint32_t v[kScanItems], local = 0, total;
  for (int k = 0; k < kScanItems; k++) {
    v[k] = base + k < n ? in[base + k] : 0u;
    local += v[k];
  }
  uint32_t run = offsets[blockIdx.x] + block_scan(local, warps, &total);
  for (int k = 0; k < kScanItems; k++) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
}

// out must hold n + 1 values; the total also goes to *total (device memory) when given.
static int exclusive_scan(const uint32_t *in, uint32_t *out, size_t n, uint32_t *total, cudaStream_t s) {
  const size_t blocks = (n + kScanThreads * kScanItems - 1) / (kScanThreads * kScanItems);
  uint32_t *sums = nullptr;
  PW_TRY(tmp_alloc(&sums, (blocks ? blocks : 1) * sizeof(uint32_t), s));
  if (blocks) scan_sums<<<(unsigned)blocks, kScanThreads, 0, s>>>(in, sums, n);
  scan_offsets<<<1, kScanThreads, 0, s>>>(sums, (uint32_t)blocks, out + n, total);
  if (blocks) scan_write<<<(unsigned)blocks, kScanThreads, 0, s>>>(in, out, sums, n);
  tmp_free(sums, s);
  return PW_OK;
}

// ------------------------------------------------------------------ raster
// The three projections (u, v, axis) of one voxelization; their columns lie one
// projection after another in the column arrays.
struct Proj { int u, v, axis; uint32_t su, sv, sa; size_t stu, stv, sta; size_t col0; };
struct Projs { Proj p[3]; };

__device__ __forceinline__ double edge_fn(const double *a, const double *b, double u, double v) {
  return (b[0] - a[0]) * (v - a[1]) - (b[1] - a[1]) * (u - a[0]);
}

__device__ __forceinline__ bool owns_edge(double value, const double *a, const double *b) {
  return value > 0 || (value == 0 && (b[1] < a[1] || (b[1] == a[1] && b[0] > a[0])));
}

// The pixels [lo, hi] of [0, size) that a triangle's extent covers, exact in
// binary32 (the coordinates' own precision); conversions saturate.
__device__ __forceinline__ void pixel_range(float a, float b, float c, uint32_t size, int *lo, uint32_t *count) {
  const int l = max(0, (int)ceilf(fminf(fminf(a, b), c)));
  const int h = (int)min((long long)size - 1, (long long)(int)floorf(fmaxf(fmaxf(a, b), c)));
  *lo = l;
  *count = h >= l ? (uint32_t)(h - l) + 1u : 0u;
}

// Counts the hits per column (FILL 0), or writes their depths: each hit takes
// the next free place of its column by counting `count` back down to zero.
// A warp takes 32 triangles: each lane finds its triangle's pixel boxes in
// binary32, and the warp then shares the boxes' pixels evenly, 32 at a time,
// with the binary64 edge functions only there.  A mesh finer than the lattice
// has few pixels per triangle (most of them none), a coarse one thousands; with
// few triangles `slices` warps share each group's pixels.  Binary64 is the
// scarce unit here (two lanes an SM and clock), and a block per triangle and
// projection, its setup in binary64, took 1.90 ms a launch on 200,000 triangles
// at 256x128x128, six launches a mesh (voxelize and create: 16.7 ms; in this
// form 4.40 ms).
// A group with more pixels than kHeavyPixels a warp is only noted here, with its place
// among all such groups' pieces, and raster_heavy shares the pieces over the GPU: a few
// large triangles in a fine mesh (a ground plate under a body) kept one warp busy while
// the others had long ended.
constexpr int kRasterThreads = 128;
constexpr uint32_t kHeavyPixels = 2048;

struct HeavyGroup {
  unsigned long long first;  // its first piece among all
  uint32_t group, proj;
};
// Notes taken so far: the groups above this bit, their pieces below it.  3 ntri / 32
// groups fit above; 2^35 pieces are 7e13 pixels.
constexpr int kHeavyBits = 35;
__host__ __device__ constexpr uint32_t heavy_groups(unsigned long long n) { return (uint32_t)(n >> kHeavyBits); }
__host__ __device__ constexpr unsigned long long heavy_pieces(unsigned long long n) {
  return n & ((1ull << kHeavyBits) - 1ull);
}

// A warp's group of triangles and their pixel boxes in one projection.
struct RasterGroup {
  float tri[32][9];
  unsigned long long first[32];  // pixels before each lane's box
  int2 corner[32];
  uint32_t width[32];
};

// Loads the lane's triangle of the group; false past the mesh's end and where a
// coordinate is not finite.
__device__ __forceinline__ bool load_triangle(const float *mesh, uint32_t ntri, uint32_t group, RasterGroup &g, float *q,
                                              uint32_t *nonfinite) {
  const uint32_t lane = threadIdx.x & 31u;
  const size_t t = (size_t)group * 32u + lane;
  bool ok = t < ntri;
#pragma unroll
  for (int k = 0; k < 9; k++) q[k] = ok ? mesh[9 * t + k] : 0.0f;
  if (ok) {
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 9; k++) finite = finite && isfinite(q[k]);
    if (!finite) {
      ok = false;
      if (nonfinite) *nonfinite = 1u;
    }
  }
#pragma unroll
  for (int k = 0; k < 9; k++) g.tri[lane][k] = q[k];
  return ok;
}

// The pixel boxes of the warp's triangles in projection p; returns their pixels' sum.
__device__ __forceinline__ unsigned long long box_triangles(const Proj &p, const float *q, bool ok, RasterGroup &g) {
  const uint32_t lane = threadIdx.x & 31u;
  const int u = p.u, v = p.v;
  const float qu[3] = {u == 0 ? q[0] : (u == 1 ? q[1] : q[2]), u == 0 ? q[3] : (u == 1 ? q[4] : q[5]),
                       u == 0 ? q[6] : (u == 1 ? q[7] : q[8])};
  const float qv[3] = {v == 0 ? q[0] : (v == 1 ? q[1] : q[2]), v == 0 ? q[3] : (v == 1 ? q[4] : q[5]),
                       v == 0 ? q[6] : (v == 1 ? q[7] : q[8])};
  int u0, v0;
  uint32_t w, h;
  pixel_range(qu[0], qu[1], qu[2], p.su, &u0, &w);
  pixel_range(qv[0], qv[1], qv[2], p.sv, &v0, &h);
  unsigned long long own = ok ? (unsigned long long)w * h : 0ull, inc = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long prev = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += prev;
  }
  const unsigned long long total = __shfl_sync(0xffffffffu, inc, 31);
  __syncwarp();
  g.first[lane] = inc - own;
  g.corner[lane] = make_int2(u0, v0);
  g.width[lane] = w;
  __syncwarp();
  return total;
}

// Pixels from, from + step, ... below `to` of the group's boxes, one a lane.
template <bool FILL>
__device__ __forceinline__ void raster_pixels(const Proj &p, const RasterGroup &g, unsigned long long from,
                                              unsigned long long to, unsigned long long step, uint32_t *count,
                                              const uint32_t *offset, double *hits) {
  const int u = p.u, v = p.v;
  for (unsigned long long k = from; k < to; k += step) {
    // the last lane whose box begins at or before pixel k
    uint32_t j = 0;
#pragma unroll
    for (uint32_t half = 16; half > 0; half >>= 1)
      if (g.first[j + half] <= k) j += half;
    const unsigned long long at = k - g.first[j];
    const uint32_t bw = g.width[j];
    const int2 c0 = g.corner[j];
    const long long pu = c0.x + (long long)(at % bw), pv = c0.y + (long long)(at / bw);
    const float *m = g.tri[j];
    const double A[3] = {m[u], m[v], m[p.axis]};
    const double B0[3] = {m[3 + u], m[3 + v], m[3 + p.axis]};
    const double C0[3] = {m[6 + u], m[6 + v], m[6 + p.axis]};
    const double signed_area = edge_fn(A, B0, C0[0], C0[1]);
    if (signed_area == 0) continue;
    const bool front = signed_area > 0;
    const double B[3] = {front ? B0[0] : C0[0], front ? B0[1] : C0[1], front ? B0[2] : C0[2]};
    const double C[3] = {front ? C0[0] : B0[0], front ? C0[1] : B0[1], front ? C0[2] : B0[2]};
    const double wa = edge_fn(B, C, (double)pu, (double)pv);
    if (!owns_edge(wa, B, C)) continue;
    const double wb = edge_fn(C, A, (double)pu, (double)pv);
    if (!owns_edge(wb, C, A)) continue;
    const double wc = edge_fn(A, B, (double)pu, (double)pv);
    if (!owns_edge(wc, A, B)) continue;
    const size_t col = p.col0 + (size_t)pu + (size_t)p.su * (size_t)pv;
    if (!FILL) {
      atomicAdd(&count[col], 1u);
    } else {
      const uint32_t place = atomicSub(&count[col], 1u) - 1u;
      hits[offset[col] + place] = (wa * A[2] + wb * B[2] + wc * C[2]) / fabs(signed_area);
    }
  }
}

template <bool FILL>
__global__ void __launch_bounds__(kRasterThreads) raster_kernel(const float *mesh, uint32_t ntri, Projs P,
                                                               uint32_t slices, uint32_t *count,
                                                               const uint32_t *offset, double *hits,
                                                               uint32_t *nonfinite, HeavyGroup *heavy,
                                                               unsigned long long *noted) {
  __shared__ RasterGroup groups[kRasterThreads / 32];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = blockIdx.x * (kRasterThreads / 32) + (threadIdx.x >> 5);
  const uint32_t group = warp / slices, slice = warp % slices;
  RasterGroup &g = groups[threadIdx.x >> 5];
  float q[9];
  const bool ok = load_triangle(mesh, ntri, group, g, q, FILL ? nullptr : nonfinite);
  for (int pr = 0; pr < 3; pr++) {
    const unsigned long long total = box_triangles(P.p[pr], q, ok, g);
    if (total > (unsigned long long)slices * kHeavyPixels) {
      if (!FILL && slice == 0u && lane == 0u) {
        const unsigned long long pieces = (total + kHeavyPixels - 1u) / kHeavyPixels;
        const unsigned long long before = atomicAdd(noted, (1ull << kHeavyBits) + pieces);
        heavy[heavy_groups(before)] = HeavyGroup{heavy_pieces(before), group, (uint32_t)pr};
      }
      continue;
    }
    raster_pixels<FILL>(P.p[pr], g, (unsigned long long)slice * 32u + lane, total, (unsigned long long)slices * 32u,
                        count, offset, hits);
  }
}

// The noted groups' pieces of kHeavyPixels, one a warp at a time (the notes lie in the
// order of their first pieces).  200,000 triangles and a ground plate of 12 at
// 512x256x256: 57 ms to voxelize with the plate's groups on a warp each, 1.6 ms so.
template <bool FILL>
__global__ void __launch_bounds__(kRasterThreads) raster_heavy(const float *mesh, uint32_t ntri, Projs P,
                                                              const HeavyGroup *heavy, uint32_t n,
                                                              unsigned long long pieces, uint32_t *count,
                                                              const uint32_t *offset, double *hits) {
  __shared__ RasterGroup groups[kRasterThreads / 32];
  const uint32_t lane = threadIdx.x & 31u;
  RasterGroup &g = groups[threadIdx.x >> 5];
  const uint64_t warps = (uint64_t)gridDim.x * (kRasterThreads / 32);
  for (uint64_t k = (uint64_t)blockIdx.x * (kRasterThreads / 32) + (threadIdx.x >> 5); k < pieces; k += warps) {
    uint32_t lo = 0, hi = n;  // the last note whose first piece is at or before piece k
    while (hi - lo > 1u) {
      const uint32_t mid = lo + (hi - lo) / 2u;
      if (heavy[mid].first <= k) lo = mid;
      else hi = mid;
    }
    const HeavyGroup note = heavy[lo];
    const Proj &p = P.p[note.proj];
    float q[9];
    const bool ok = load_triangle(mesh, ntri, note.group, g, q, nullptr);
    const unsigned long long total = box_triangles(p, q, ok, g);
    const unsigned long long from = (k - note.first) * kHeavyPixels;
    raster_pixels<FILL>(p, g, from + lane, min(total, from + kHeavyPixels), 32u, count, offset, hits);
    __syncwarp();  // the group's words are free again
  }
}

// Sorts each column's hits and adds its spans [ceil(h0), ceil(h1)) to the votes, the
// projections side by side (blockIdx.y): a vote is one added to its byte of a word, and
// nothing waits for the sum: 8 us at 256x128x128 (a load, an increment and a store a
// cell, one projection after another, took 82 us, each lane waiting for its last cell).
// Threads run over the columns with x the fastest of (u, v); columns along x are filled
// by the whole warp, one lane's span at a time, a word of four cells a lane.
__device__ __forceinline__ void add_vote(uint32_t *votes, size_t cell) {
  atomicAdd(&votes[cell >> 2], 1u << (8u * (uint32_t)(cell & 3u)));
}

__global__ void __launch_bounds__(128) column_kernel(Projs projs, const uint32_t *offset, double *hits,
                                                     uint32_t *votes, uint32_t *odd) {
  const Proj &P = projs.p[blockIdx.y];
  const size_t ncol = (size_t)P.su * P.sv, id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if ((size_t)blockIdx.x * blockDim.x >= ncol) return;
  const uint32_t lane = threadIdx.x & 31u;
  const bool along_x = P.axis == 0, v_is_x = P.v == 0;
  uint32_t u = 0, v = 0, n = 0, at = 0;
  if (id < ncol) {
    u = v_is_x ? (uint32_t)(id / P.sv) : (uint32_t)(id % P.su);
    v = v_is_x ? (uint32_t)(id % P.sv) : (uint32_t)(id / P.su);
    const size_t col = P.col0 + (size_t)u + (size_t)P.su * v;
    at = offset[col];
    n = offset[col + 1] - at;
  }
  double *h = hits + at;
  for (uint32_t i = 1; i < n; i++) {  // insertion sort: columns hold few hits
    double key = h[i];
    int j = (int)i - 1;
    while (j >= 0 && h[j] > key) { h[j + 1] = h[j]; j--; }
    h[j + 1] = key;
  }
  if (n % 2) *odd = 1u;
  const size_t base = (size_t)u * P.stu + (size_t)v * P.stv;
  for (uint32_t pair = 0; __any_sync(0xffffffffu, pair + 1 < n); pair += 2) {
    long long s0 = 0, s1 = 0;
    if (pair + 1 < n) {
      s0 = (long long)fmax(0.0, ceil(h[pair]));
      s1 = (long long)fmin((double)P.sa, ceil(h[pair + 1]));
    }
    if (!along_x) {
      for (long long c = s0; c < s1; c++) add_vote(votes, base + (size_t)c * P.sta);
      continue;
    }
    for (uint32_t left = __ballot_sync(0xffffffffu, s0 < s1); left; left &= left - 1u) {
      const int src = __ffs(left) - 1;
      const long long a = __shfl_sync(0xffffffffu, s0, src), b = __shfl_sync(0xffffffffu, s1, src);
      const size_t row = __shfl_sync(0xffffffffu, (unsigned long long)base, src);
      const size_t from = row + (size_t)a, to = row + (size_t)b;  // cells, a word of four a lane
      for (size_t w = (from >> 2) + lane; w <= (to - 1) >> 2; w += 32) {
        uint32_t add = 0x01010101u;
        if (4 * w < from) add &= 0xffffffffu << (8u * (uint32_t)(from - 4 * w));
        if (4 * w + 4 > to) add &= 0xffffffffu >> (8u * (uint32_t)(4 * w + 4 - to));
        atomicAdd(&votes[w], add);
      }
    }
  }
}

// Every cell's kind from the meshes' votes (two of the three projections; body
// before supports), then the boundary planes (voxelize.ts:123-135: the floor
// plane, the top plane over a floor, the x faces), and countCells
// (voxelize.ts:137-154): solid cells, and the (y, z) rows that hold one.
// body or sup is null without such a mesh.
__global__ void kinds_kernel(const uint8_t *body, const uint8_t *sup, uint32_t *flags, uint32_t nx, uint32_t ny,
                             uint32_t nz, int floor_on, uint32_t *solid, uint8_t *body_rows, uint8_t *wall_rows) {
  const size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = at < (size_t)nx * ny * nz;
  const uint32_t i = (uint32_t)at, row = i / nx, x = i - row * nx, z = row / ny;
  uint32_t t = pw::FLUID;
  if (in) {
    if (body && body[at] >= 2) t = pw::SOLID;
    else if (sup && sup[at] >= 2) t = pw::SUPPORT;
    if (floor_on && z == 0) t = pw::FLOOR;
    else if (floor_on && z == nz - 1) t = pw::EQ;
    else if (x == 0 || x == nx - 1) t = pw::EQ;
    flags[at] = t;
    if (t == pw::SOLID) body_rows[row] = 1;
    if (t == pw::SOLID || t == pw::SUPPORT) wall_rows[row] = 1;
  }
  const uint32_t n = __popc(__ballot_sync(0xffffffffu, in && t == pw::SOLID));
  if (n && (threadIdx.x & 31u) == 0u) atomicAdd(solid, n);
}

// The rows marked in each of the two row arrays (one after the other) into out[0] and out[1].
__global__ void sum_rows_kernel(const uint8_t *v, size_t rows, uint32_t *out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
  for (int a = 0; a < 2; a++) {
    const uint32_t n = __popc(__ballot_sync(0xffffffffu, i < rows && v[(size_t)a * rows + i] != 0));
    if (n && (threadIdx.x & 31u) == 0u) atomicAdd(out + a, n);
  }
}

// markWalls, wall-links.ts:34-51, gathered per fluid cell: bit (3+i) when the
// pull source x - c_i (x bounded, y periodic, z bounded with a floor) is a wall.
// Only fluid words change and their type bits stay, so concurrent readers of a
// neighbour's type see the same kind before and after its write.  Fluid cells
// next to the body also get kBodyBit, until pack_links_kernel takes it out.
// Each block sums the links and the body's neighbours of its 1,024 cells, all
// that the packing pass needs of the cells before its own: with 32-bit cell
// arithmetic and no per-cell counts this pass, the packing pass and their scan
// take the place of six passes (134 us for the masks alone, with 64-bit
// remainders, and 103 us for the counts' scans, the q offsets, the fractions
// and the boundary list, at 256x128x128).  Where none of the nine rows around a cell
// holds a wall (wall_rows, the same bytes for a whole warp) its 18 neighbours are not
// read.
constexpr uint32_t kBodyBit = 1u << 31;
constexpr uint32_t kLinkBits = 0x3ffff0u;
constexpr int kMaskThreads = 256, kMaskCells = 4 * kMaskThreads;

__global__ void __launch_bounds__(kMaskThreads) wall_mask_kernel(uint32_t *flags, uint32_t nx, uint32_t ny, uint32_t nz,
                                                                int floor_on, const uint8_t *wall_rows, uint32_t *sums,
                                                                uint32_t blocks) {
  __shared__ uint32_t total[2];
  if (threadIdx.x < 2) total[threadIdx.x] = 0u;
  __syncthreads();
  const size_t cells = (size_t)nx * ny * nz, base = (size_t)blockIdx.x * kMaskCells + threadIdx.x;
  const uint32_t plane = nx * ny;
  uint32_t links = 0, next = 0;
  for (int k = 0; k < 4; k++) {
    const size_t at = base + (size_t)k * kMaskThreads;
    if (at >= cells) break;
    const uint32_t i = (uint32_t)at, f = flags[at];
    if ((f & 7u) != pw::FLUID) continue;
    const uint32_t row = i / nx, x = i - row * nx, z = row / ny, y = row - z * ny;
    const uint32_t rm = y == 0 ? ny - 1 : y - 1, rp = y + 1 == ny ? 0 : y + 1;
    const uint32_t pm = (z == 0 ? nz - 1 : z - 1) * ny, p0 = z * ny, pp = (z + 1 == nz ? 0 : z + 1) * ny;
    uint32_t walls = wall_rows[pm + rm] | wall_rows[pm + y] | wall_rows[pm + rp] | wall_rows[p0 + rm] | wall_rows[row] |
                     wall_rows[p0 + rp] | wall_rows[pp + rm] | wall_rows[pp + y] | wall_rows[pp + rp];
    if (!walls && !(floor_on && z <= 1u)) continue;
    // offsets to the source of each axis' step (mod 2^32, as the cell index)
    const uint32_t ym = y == 0 ? plane - nx : 0u - nx, yp = y + 1 == ny ? nx - plane : nx;
    const uint32_t span = plane * nz;
    const uint32_t zm = z == 0 ? span - plane : 0u - plane, zp = z + 1 == nz ? plane - span : plane;
    const bool has_xm = x > 0, has_xp = x + 1 < nx, has_zm = !(floor_on && z == 0), has_zp = !(floor_on && z + 1 == nz);
    uint32_t mask = 0;
    bool body = false;
#pragma unroll
    for (int d = 1; d < 19; d++) {
      const int cx = pw::cx_of(d), cy = pw::cy_of(d), cz = pw::cz_of(d);
      if ((cx > 0 && !has_xm) || (cx < 0 && !has_xp) || (cz > 0 && !has_zm) || (cz < 0 && !has_zp)) continue;
      const uint32_t src = i + (cx > 0 ? ~0u : (cx < 0 ? 1u : 0u)) + (cy > 0 ? ym : (cy < 0 ? yp : 0u)) +
                           (cz > 0 ? zm : (cz < 0 ? zp : 0u));
      const uint32_t t = flags[src] & 7u;
      if (t >= pw::SOLID && t <= pw::FLOOR) mask |= 1u << (3 + d);
      body = body || t == pw::SOLID;
    }
    if (mask) flags[at] = f | mask | (body ? kBodyBit : 0u);
    links += __popc(mask);
    next += body ? 1u : 0u;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    links += __shfl_down_sync(0xffffffffu, links, o);
    next += __shfl_down_sync(0xffffffffu, next, o);
  }
  if ((threadIdx.x & 31u) == 0u && links) {
    atomicAdd(&total[0], links);
    atomicAdd(&total[1], next);
  }
  __syncthreads();
  if (threadIdx.x < 2) sums[(size_t)threadIdx.x * blocks + blockIdx.x] = total[threadIdx.x];
}

// The packed geometry of a block's 1,024 cells: q offsets, halfway fractions and
// the ascending list of the body's neighbours, from the block's offsets; with
// links also every link's cell and direction, in the fractions' order.
__global__ void __launch_bounds__(kMaskThreads) pack_links_kernel(uint32_t *flags, size_t cells, const uint32_t *offsets,
                                                                 uint32_t blocks, uint32_t *qoff, float *fractions,
                                                                 uint32_t *boundary, uint2 *links) {
  __shared__ uint32_t warps[33];
  uint32_t at_link = offsets[blockIdx.x], at_body = offsets[(size_t)blocks + blockIdx.x];
  for (int k = 0; k < 4; k++) {
    const size_t i = (size_t)blockIdx.x * kMaskCells + (size_t)k * kMaskThreads + threadIdx.x;
    const uint32_t f = i < cells ? flags[i] : 0u;
    const uint32_t n = __popc(f & kLinkBits), b = f >> 31;
    uint32_t off = PW_NO_Q;
    if (__syncthreads_or(n)) {
      uint32_t sum_n, sum_b;
      const uint32_t first = at_link + block_scan(n, warps, &sum_n);
      __syncthreads();
      const uint32_t rank = at_body + block_scan(b, warps, &sum_b);
      if (n) {
        off = first;
        for (uint32_t r = 0; r < n; r++) fractions[first + r] = 0.5f;
        if (links) {
          uint32_t r = first;
          for (uint32_t m = f & kLinkBits; m; m &= m - 1u) links[r++] = make_uint2((uint32_t)i, (uint32_t)__ffs(m) - 4u);
        }
        if (b) {
          boundary[rank] = (uint32_t)i;
          flags[i] = f & ~kBodyBit;
        }
      }
      at_link += sum_n;
      at_body += sum_b;
    }
    if (i < cells) qoff[i] = off;
  }
}

static inline unsigned nblk(size_t n, unsigned b = 256) { return (unsigned)((n + b - 1) / b); }

// What the voxelization's kernels report, one copy to the host.
struct GridInfo {
  uint32_t solid, frontal, blocked;  // countCells
  uint32_t odd[2];                   // body, supports: a column with an odd number of hits (an open mesh)
  uint32_t nonfinite;                // a coordinate that is not finite
  uint32_t hits;
  uint32_t links, boundary;          // wall links; fluid cells next to the body
  uint32_t missed;                   // links whose cast met no triangle
  unsigned long long heavy[2];       // body, supports: the raster's notes (kHeavyBits)
};

static int read_info(const GridInfo *info, GridInfo *out, cudaStream_t s) {
  PW_TRY(cudaMemcpyAsync(out, info, sizeof(GridInfo), cudaMemcpyDeviceToHost, s));
  PW_TRY(cudaStreamSynchronize(s));
  return PW_OK;
}

// The votes of one mesh, one byte a cell (null without triangles; the caller's to
// free).  which: 0 the body, 1 the supports.
static int vote_mesh(const float *d_mesh, uint32_t ntri, uint32_t nx, uint32_t ny, uint32_t nz, int which,
                     GridInfo *info, uint8_t **votes_out, cudaStream_t s) {
  if (ntri == 0) return PW_OK;
  const size_t cells = (size_t)nx * ny * nz;
  const uint32_t sizes[3] = {nx, ny, nz};
  const size_t strides[3] = {1, nx, (size_t)nx * ny};
  const int PROJS[3][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}};
  Projs P;
  size_t ncol = 0;
  for (int p = 0; p < 3; p++) {
    const int u = PROJS[p][0], v = PROJS[p][1], a = PROJS[p][2];
    P.p[p] = Proj{u, v, a, sizes[u], sizes[v], sizes[a], strides[u], strides[v], strides[a], ncol};
    ncol += (size_t)sizes[u] * sizes[v];
  }
  GridInfo got{};
  double *hits = nullptr;
  // one warp a group of 32 triangles, or as many as fill the SMs with 16
  const uint32_t groups = (ntri + 31u) / 32u;
  cudaError_t e = tmp_alloc(votes_out, (cells + 3) / 4 * 4, s);
  uint8_t *votes = *votes_out;
  // the notes, the columns' counts and offsets in one allocation
  const size_t notes = 3 * (size_t)groups * sizeof(HeavyGroup);
  char *columns = nullptr;
  if (e == cudaSuccess) e = tmp_alloc(&columns, notes + (2 * ncol + 1) * 4, s);
  HeavyGroup *heavy = reinterpret_cast<HeavyGroup *>(columns);
  uint32_t *count = reinterpret_cast<uint32_t *>(columns + notes), *offset = count + ncol;
  int rc = e == cudaSuccess ? PW_OK : cuda_status(e, "voxelize columns");
  const uint32_t slices = std::max(1u, std::min(1024u, multiprocessors() * 16u / groups));
  const unsigned rblocks = (unsigned)(((uint64_t)groups * slices + kRasterThreads / 32 - 1) / (kRasterThreads / 32));
  if (rc == PW_OK) {
    cudaMemsetAsync(votes, 0, (cells + 3) / 4 * 4, s);
    cudaMemsetAsync(count, 0, ncol * 4, s);
    raster_kernel<false><<<rblocks, kRasterThreads, 0, s>>>(d_mesh, ntri, P, slices, count, nullptr, nullptr,
                                                            &info->nonfinite, heavy, &info->heavy[which]);
    rc = exclusive_scan(count, offset, ncol, &info->hits, s);
  }
  if (rc == PW_OK) rc = read_info(info, &got, s);
  const uint32_t noted = heavy_groups(got.heavy[which]);
  const unsigned long long pieces = heavy_pieces(got.heavy[which]);
  const unsigned hblocks = (unsigned)std::min<unsigned long long>((pieces + kRasterThreads / 32 - 1) / (kRasterThreads / 32),
                                                                  16ull * multiprocessors());
  if (rc == PW_OK && noted && !got.nonfinite) {  // their hits too, and the columns' offsets anew
    raster_heavy<false><<<hblocks, kRasterThreads, 0, s>>>(d_mesh, ntri, P, heavy, noted, pieces, count, nullptr,
                                                           nullptr);
    rc = exclusive_scan(count, offset, ncol, &info->hits, s);
    if (rc == PW_OK) rc = read_info(info, &got, s);
  }
  if (rc == PW_OK && got.nonfinite) {
    set_error("Mesh coordinates must be finite.");
    rc = PW_ERR_INVALID;
  }
  if (rc == PW_OK && got.hits) {
    e = tmp_alloc(&hits, (size_t)got.hits * sizeof(double), s);
    if (e != cudaSuccess) rc = cuda_status(e, "voxelize hits");
    if (rc == PW_OK) {
      raster_kernel<true><<<rblocks, kRasterThreads, 0, s>>>(d_mesh, ntri, P, slices, count, offset, hits, nullptr,
                                                             nullptr, nullptr);
      if (noted)
        raster_heavy<true><<<hblocks, kRasterThreads, 0, s>>>(d_mesh, ntri, P, heavy, noted, pieces, count, offset,
                                                              hits);
      size_t most = 0;
      for (int p = 0; p < 3; p++) most = std::max(most, (size_t)P.p[p].su * P.p[p].sv);
      column_kernel<<<dim3(nblk(most, 128), 3), 128, 0, s>>>(P, offset, hits, reinterpret_cast<uint32_t *>(votes),
                                                             &info->odd[which]);
    }
  }
  tmp_free(columns, s); tmp_free(hits, s);
  return rc;
}

// ------------------------------------------------------------------ link fractions
// binTriangles / nearestLinkHit / intersection (src/geometry/triangle-bins.ts:1-162)
// and linkFraction (src/geometry/wall-links.ts:53-80) in binary64: four-cell bins
// of triangles, then each wall link's segment from the cell centre toward the wall
// against the triangles of its bins, nearest Moller-Trumbore hit kept.  The minimum
// does not depend on the order of a bin's items, so bins fill with atomics and the
// fractions match the sequential reference bit for bit.
constexpr int kBin = 4;

struct DevBins {
  const float *mesh = nullptr;
  float *bounds = nullptr;      // 6 per triangle: float lo, hi
  uint32_t *start = nullptr;    // nbins + 1
  uint32_t *items = nullptr;    // triangle per entry
  int bx = 0, by = 0, bz = 0;
};

__device__ __forceinline__ void bin_range(const double *lo, const double *hi, const DevBins &B, long *r) {
  const int dims[3] = {B.bx, B.by, B.bz};
  for (int a = 0; a < 3; a++) {
    long mn = (long)floor(lo[a] / kBin), mx = (long)floor(hi[a] / kBin);
    r[2 * a] = mn < 0 ? 0 : mn;
    r[2 * a + 1] = mx > dims[a] - 1 ? dims[a] - 1 : mx;
  }
}

// pass 0 counts the bins each triangle's box touches, pass 1 files the triangle.
__global__ void bin_triangles_kernel(DevBins B, uint32_t ntri, uint32_t *count, int pass) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntri) return;
  const float *p = B.mesh + 9 * (size_t)t;
  double lo[3], hi[3];
  for (int a = 0; a < 3; a++) {
    double x = p[a], y = p[a + 3], z = p[a + 6];
    lo[a] = fmin(fmin(x, y), z);
    hi[a] = fmax(fmax(x, y), z);
  }
  if (pass == 0)
    for (int a = 0; a < 3; a++) { B.bounds[6 * t + a] = (float)lo[a]; B.bounds[6 * t + 3 + a] = (float)hi[a]; }
  long r[6];
  bin_range(lo, hi, B, r);
  for (long z = r[4]; z <= r[5]; z++)
    for (long y = r[2]; y <= r[3]; y++)
      for (long x = r[0]; x <= r[1]; x++) {
        size_t k = (size_t)x + (size_t)B.bx * ((size_t)y + (size_t)B.by * (size_t)z);
        uint32_t slot = atomicAdd(&count[k], 1u);
        if (pass == 1) B.items[B.start[k] + slot] = t;
      }
}

// intersection, triangle-bins.ts:60-94: the hit depth t along d, or false.  A u or v that
// the test must refuse, by more than EPS (far beyond the rounding), is refused before the
// division: binary64 divisions are most of a test's time.  u lies in [-EPS, 1 + EPS], but v
// may reach 1 + 2 EPS, beside u = -EPS.
__device__ __forceinline__ bool segment_hit(const float *p, const double *o, const double *d, double *t) {
  const double EPS = 1e-9;
  double ax = p[0], ay = p[1], az = p[2];
  double e1x = (double)p[3] - ax, e1y = (double)p[4] - ay, e1z = (double)p[5] - az;
  double e2x = (double)p[6] - ax, e2y = (double)p[7] - ay, e2z = (double)p[8] - az;
  double px = d[1] * e2z - d[2] * e2y;
  double py = d[2] * e2x - d[0] * e2z;
  double pz = d[0] * e2y - d[1] * e2x;
  double det = e1x * px + e1y * py + e1z * pz;
  if (fabs(det) < 2.220446049250313e-16) return false;
  const auto outside = [&](double num) {
    const double n = det < 0 ? -num : num, a = fabs(det);
    return n < -2 * EPS * a || n > (1 + 3 * EPS) * a;
  };
  double tx = o[0] - ax, ty = o[1] - ay, tz = o[2] - az;
  double un = tx * px + ty * py + tz * pz;
  if (outside(un)) return false;
  double u = un / det;
  if (u < -EPS || u > 1 + EPS) return false;
  double qx = ty * e1z - tz * e1y;
  double qy = tz * e1x - tx * e1z;
  double qz = tx * e1y - ty * e1x;
  double vn = d[0] * qx + d[1] * qy + d[2] * qz;
  if (outside(vn)) return false;
  double v = vn / det;
  if (v < -EPS || u + v > 1 + EPS) return false;
  double tt = (e2x * qx + e2y * qy + e2z * qz) / det;
  if (tt >= -EPS && tt <= 1 + EPS) { *t = tt; return true; }
  return false;
}

// A double's bits in the order of its value.
__device__ __forceinline__ unsigned long long ordered(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b >> 63 ? ~b : b | 1ull << 63;
}
__device__ __forceinline__ double from_ordered(unsigned long long k) {
  return __longlong_as_double((long long)(k >> 63 ? k & ~(1ull << 63) : ~k));
}

// linkFraction of every wall link: FLOOR links keep 1/2; SOLID links cast against
// the body, SUPPORT links against the supports; a miss keeps 1/2 and counts; hits
// clamp to [1e-3, 1].
// A warp takes eight consecutive links, which share most of their bins.  For one
// link after another all lanes scan its bins' triangles (nearestLinkHit,
// triangle-bins.ts:136-161; bins next to each other in x are one range) with the
// box test in binary32: the segment's ends are whole numbers, rounded toward the
// test's inside, so it decides as binary64 does.  The few triangles that pass go
// to a queue, and the binary64 intersections run for 32 queued pairs at a time:
// binary64 issues at the same rate for one lane as for 32.  A thread per cell
// with its links and triangles in turn took 4.92 ms for the 70,000 links of a
// 150x75x61 grid with 12,288 triangles (14,000 of them cast, the others on the floor).
// With 32 links a warp there were too few warps to cover the loads (210 us); eight take
// 92 us.
constexpr int kLinkThreads = 128;
constexpr uint32_t kWarpLinks = 8;
struct LinkCast { int ox, oy, oz, dir; };
__global__ void __launch_bounds__(kLinkThreads) link_fraction_kernel(const uint32_t *flags, const uint2 *links,
                                                                    uint32_t nlinks, float *fractions, uint32_t nx,
                                                                    uint32_t ny, uint32_t nz, DevBins body, DevBins sup,
                                                                    int has_sup, uint32_t *missed) {
  __shared__ LinkCast cast[kLinkThreads / 32][32];
  __shared__ unsigned long long best[kLinkThreads / 32][32];
  __shared__ uint2 queue[kLinkThreads / 32][64];  // (triangle, link's lane), bit 5 of the lane: the supports
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint32_t first = (blockIdx.x * (kLinkThreads / 32) + w) * kWarpLinks;
  if (first >= nlinks) return;  // the whole warp
  const uint32_t link = lane < kWarpLinks ? first + lane : nlinks;
  uint32_t target = 0;  // 1 the body, 2 the supports: this lane's link is cast
  LinkCast c = {0, 0, 0, 0};
  bool hit = link < nlinks;  // until a cast misses
  if (link < nlinks) {
    const uint2 l = links[link];
    const uint32_t row = l.x / nx, x = l.x - row * nx, z = row / ny, y = row - z * ny;
    const int i = (int)l.y, cx = pw::cx_of(i), cy = pw::cy_of(i), cz = pw::cz_of(i);
    // the wall x - c_i: x bounded, y periodic, z periodic unless a floor bounds it
    const long wx = (long)x - cx, wy = ((long)y - cy + (long)ny) % (long)ny, wz = ((long)z - cz + (long)nz) % (long)nz;
    const uint32_t type = flags[(size_t)wx + (size_t)nx * ((size_t)wy + (size_t)ny * (size_t)wz)] & 7u;
    if (type != pw::FLOOR) {
      target = type != pw::SUPPORT ? 1u : (has_sup ? 2u : 0u);
      hit = false;
    }
    c = LinkCast{(int)(wx + cx), (int)(wy + cy), (int)(wz + cz), i};
  }
  const unsigned long long none = ordered(CUDART_INF);
  cast[w][lane] = c;
  best[w][lane] = none;
  __syncwarp();
  uint32_t queued = 0;
  const auto flush = [&](uint32_t n) {  // the first n queued pairs (n <= 32)
    __syncwarp();
    if (lane < n) {
      const uint2 e = queue[w][lane];
      const LinkCast k = cast[w][e.y & 31u];
      const double o[3] = {(double)k.ox, (double)k.oy, (double)k.oz};
      const double d[3] = {(double)-pw::cx_of(k.dir), (double)-pw::cy_of(k.dir), (double)-pw::cz_of(k.dir)};
      double t;
      if (segment_hit((e.y & 32u ? sup.mesh : body.mesh) + 9 * (size_t)e.x, o, d, &t))
        atomicMin(&best[w][e.y & 31u], ordered(t));
    }
    __syncwarp();
  };
  for (uint32_t todo = __ballot_sync(0xffffffffu, target != 0u); todo; todo &= todo - 1u) {
    const uint32_t j = (uint32_t)__ffs(todo) - 1u;
    const LinkCast k = cast[w][j];
    const bool in_sup = __shfl_sync(0xffffffffu, target, (int)j) == 2u;
    const DevBins &B = in_sup ? sup : body;
    const int o[3] = {k.ox, k.oy, k.oz};
    const int d[3] = {-pw::cx_of(k.dir), -pw::cy_of(k.dir), -pw::cz_of(k.dir)};
    const int dims[3] = {B.bx, B.by, B.bz};
    float lo[3], hi[3];
    int r[6];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int mn = min(o[a], o[a] + d[a]), mx = max(o[a], o[a] + d[a]);
      lo[a] = __int2float_ru(mn);
      hi[a] = __int2float_rd(mx);
      r[2 * a] = max(mn >> 2, 0);
      r[2 * a + 1] = min(mx >> 2, dims[a] - 1);
    }
    if (r[0] > r[1]) continue;
    for (int bz = r[4]; bz <= r[5]; bz++)
      for (int by = r[2]; by <= r[3]; by++) {
        const size_t row = (size_t)B.bx * ((size_t)by + (size_t)B.by * (size_t)bz);
        const uint32_t end = B.start[row + (size_t)r[1] + 1];
        for (uint32_t it = B.start[row + (size_t)r[0]]; it < end; it += 32u) {
          uint32_t tri = 0;
          bool near = false;
          if (it + lane < end) {
            tri = B.items[it + lane];
            const float *bd = B.bounds + 6 * (size_t)tri;
            near = bd[0] <= hi[0] && bd[3] >= lo[0] && bd[1] <= hi[1] && bd[4] >= lo[1] && bd[2] <= hi[2] &&
                   bd[5] >= lo[2];
          }
          const uint32_t m = __ballot_sync(0xffffffffu, near);
          if (!m) continue;
          if (near) queue[w][queued + __popc(m & ((1u << lane) - 1u))] = make_uint2(tri, j | (in_sup ? 32u : 0u));
          queued += __popc(m);
          if (queued >= 32u) {
            flush(32u);
            queued -= 32u;
            const uint2 rest = queue[w][32u + lane];
            __syncwarp();
            if (lane < queued) queue[w][lane] = rest;
          }
        }
      }
  }
  flush(queued);
  double q = 0.5;
  if (best[w][lane] != none) {
    hit = true;
    q = from_ordered(best[w][lane]);
  }
  const uint32_t misses = __popc(__ballot_sync(0xffffffffu, link < nlinks && !hit));
  if (misses && lane == 0u) atomicAdd(missed, misses);
  if (link < nlinks) {
    double f = q < 1 ? q : 1;
    f = f > 1e-3 ? f : 1e-3;
    fractions[link] = (float)f;
  }
}

static void free_bins(DevBins &B, cudaStream_t s) {
  tmp_free(B.bounds, s); tmp_free(B.start, s); tmp_free(B.items, s);
  B = DevBins();
}

static int build_bins(const float *d_mesh, uint32_t ntri, uint32_t nx, uint32_t ny, uint32_t nz, DevBins *out,
                      cudaStream_t s) {
  DevBins B;
  B.mesh = d_mesh;
  B.bx = (int)((nx + kBin - 1) / kBin); B.by = (int)((ny + kBin - 1) / kBin); B.bz = (int)((nz + kBin - 1) / kBin);
  size_t nb = (size_t)B.bx * B.by * B.bz;
  uint32_t *count = nullptr, total = 0;
  cudaError_t e = tmp_alloc(&B.bounds, (ntri ? ntri : 1) * 6 * sizeof(float), s);
  if (e == cudaSuccess) e = tmp_alloc(&B.start, (nb + 1) * 4, s);
  if (e == cudaSuccess) e = tmp_alloc(&count, nb * 4, s);
  int rc = e == cudaSuccess ? PW_OK : cuda_status(e, "triangle bins");
  if (rc == PW_OK) {
    cudaMemsetAsync(count, 0, nb * 4, s);
    if (ntri) bin_triangles_kernel<<<nblk(ntri, 128), 128, 0, s>>>(B, ntri, count, 0);
    rc = exclusive_scan(count, B.start, nb, nullptr, s);
  }
  if (rc == PW_OK) {
    e = cudaMemcpyAsync(&total, B.start + nb, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = tmp_alloc(&B.items, ((size_t)total ? total : 1) * 4, s);
    if (e != cudaSuccess) rc = cuda_status(e, "triangle bins");
  }
  if (rc == PW_OK) {
    cudaMemsetAsync(count, 0, nb * 4, s);
    if (ntri) bin_triangles_kernel<<<nblk(ntri, 128), 128, 0, s>>>(B, ntri, count, 1);
  }
  tmp_free(count, s);
  if (rc != PW_OK) { free_bins(B, s); return rc; }
  *out = B;
  return PW_OK;
}

// Measured fractions for every wall link of a finished grid (buildWallLinks with
// measureFractions, wall-links.ts:99-131); sets stats.missed_links.
static int measure_links(pw_grid *g, const float *d_body, uint32_t nbody, const float *d_sup, uint32_t nsup,
                         bool has_sup, const uint2 *links, GridInfo *info, cudaStream_t s) {
  DevBins body, sup;
  GridInfo got{};
  int rc = build_bins(d_body, nbody, g->nx, g->ny, g->nz, &body, s);
  if (rc == PW_OK && has_sup) rc = build_bins(d_sup, nsup, g->nx, g->ny, g->nz, &sup, s);
  if (rc == PW_OK) {
    const uint32_t n = (uint32_t)g->nfrac;
    link_fraction_kernel<<<nblk(n, kWarpLinks * (kLinkThreads / 32)), kLinkThreads, 0, s>>>(g->flags, links, n, g->fractions, g->nx, g->ny,
                                                                        g->nz, body, sup, has_sup ? 1 : 0, &info->missed);
    rc = read_info(info, &got, s);
  }
  free_bins(body, s);
  free_bins(sup, s);
  if (rc == PW_OK) g->stats.missed_links = got.missed;
  return rc;
}

static bool finite_mesh(const float *m, uint32_t ntri) {
  for (size_t k = 0; k < 9 * (size_t)ntri; k++)
    if (!std::isfinite(m[k])) return false;
  return true;
}

// From the meshes' votes to the finished grid: kinds, wall masks, q offsets,
// halfway fractions, boundary list, counts; with links_out also the list of the
// links (the caller's to free).
static int finish_grid(pw_grid *g, const uint8_t *body, const uint8_t *sup, int floor_on, GridInfo *info,
                       uint2 **links_out, cudaStream_t s) {
  const size_t cells = g->cells, rows = (size_t)g->ny * g->nz;
  const uint32_t blocks = nblk(cells, kMaskCells);
  uint32_t *sums = nullptr;
  uint8_t *marked = nullptr;
  GridInfo got{};
  cudaError_t e = tmp_alloc(&sums, 2 * (size_t)blocks * 4, s);
  if (e == cudaSuccess) e = tmp_alloc(&marked, 2 * rows, s);
  int rc = e == cudaSuccess ? PW_OK : cuda_status(e, "voxelize counts");
  if (rc == PW_OK) {
    cudaMemsetAsync(marked, 0, 2 * rows, s);
    kinds_kernel<<<nblk(cells), 256, 0, s>>>(body, sup, g->flags, g->nx, g->ny, g->nz, floor_on, &info->solid, marked,
                                             marked + rows);
    sum_rows_kernel<<<nblk(rows), 256, 0, s>>>(marked, rows, &info->frontal);
    wall_mask_kernel<<<blocks, kMaskThreads, 0, s>>>(g->flags, g->nx, g->ny, g->nz, floor_on, marked + rows, sums, blocks);
    scan_offsets<<<2, kScanThreads, 0, s>>>(sums, blocks, &info->links, nullptr);
    rc = read_info(info, &got, s);
  }
  if (rc == PW_OK) {
    Arena a;
    a.want((void **)&g->fractions, (size_t)got.links * 4);
    a.want((void **)&g->boundary, (size_t)got.boundary * 4);
    e = a.alloc(&g->link_arrays);
    if (e == cudaSuccess && links_out && got.links) e = tmp_alloc(links_out, (size_t)got.links * sizeof(uint2), s);
    if (e != cudaSuccess) rc = cuda_status(e, "voxelize links");
  }
  if (rc == PW_OK) {
    pack_links_kernel<<<blocks, kMaskThreads, 0, s>>>(g->flags, cells, sums, blocks, g->qoff, g->fractions,
                                                      g->boundary, links_out ? *links_out : nullptr);
    e = cudaGetLastError();
    if (e != cudaSuccess) rc = cuda_status(e, "voxelize finish");
  }
  tmp_free(sums, s); tmp_free(marked, s);
  if (rc != PW_OK) return rc;
  g->nfrac = got.links;
  g->nboundary = got.boundary;
  pw_grid_stats &st = g->stats;
  st.nx = g->nx; st.ny = g->ny; st.nz = g->nz;
  st.solid_cells = got.solid;
  st.frontal_cells = got.frontal;
  st.blockage = (double)got.blocked / ((double)g->ny * g->nz);
  st.watertight = !got.odd[0] && !got.odd[1];
  st.missed_links = 0;
  st.geometry_len = 2 * (uint64_t)cells + g->nfrac;
  st.boundary_cells = g->nboundary;
  return PW_OK;
}

// ------------------------------------------------------------------ validation
// validateGeometry's mask rule (geometry-contract.ts:20-58) with every axis
// periodic: non-fluid cells carry their kind alone, fluid cells exactly the
// walls among their wrapped pull sources.
__global__ void validate_kernel(const uint32_t *flags, uint32_t nx, uint32_t ny, uint32_t nz,
                                unsigned long long *first_bad) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t cells = (size_t)nx * ny * nz;
  if (i >= cells) return;
  uint32_t f = flags[i], kind = f & 7u;
  uint32_t expected = 0;
  if (kind == pw::FLUID) {
    long x = (long)(i % nx), y = (long)((i / nx) % ny), z = (long)(i / ((size_t)nx * ny));
#pragma unroll
    for (int d = 1; d < 19; d++) {
      long sx = (x - pw::cx_of(d) + nx) % nx, sy = (y - pw::cy_of(d) + ny) % ny, sz = (z - pw::cz_of(d) + nz) % nz;
      uint32_t t = flags[(size_t)sx + (size_t)nx * ((size_t)sy + (size_t)ny * (size_t)sz)] & 7u;
      if (t >= pw::SOLID && t <= pw::FLOOR) expected |= 1u << (3 + d);
    }
  }
  if (kind > pw::EQ || f != (kind | expected)) atomicMin(first_bad, (unsigned long long)i);
}

}  // namespace pwhost

using namespace pwhost;

extern "C" {

const char *pw_last_error(void) { return pwhost::last_error(); }
const char *pw_version(void) { return "pocketwind_gb300 0.1 (sm_103a)"; }

int pw_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) { cudaGetLastError(); return 0; }
  return n;
}

int pw_voxelize(const float *body, uint32_t body_triangles, const float *supports,
                uint32_t support_triangles, uint32_t nx, uint32_t ny, uint32_t nz, int floor_on,
                pw_grid **out) {
  return pw_voxelize_opts(body, body_triangles, supports, support_triangles, nx, ny, nz, floor_on, 0, out);
}

int pw_voxelize_opts(const float *body, uint32_t body_triangles, const float *supports,
                     uint32_t support_triangles, uint32_t nx, uint32_t ny, uint32_t nz, int floor_on,
                     int link_fractions, pw_grid **out) {
  if (!out) { set_error("out is NULL"); return PW_ERR_INVALID; }
  *out = nullptr;
  if (nx < 2 || ny < 2 || nz < 2) {
    set_error("Grid dimensions must be integers of at least two cells.");
    return PW_ERR_INVALID;
  }
  size_t cells = (size_t)nx * ny * nz;
  if (cells > 0xffffffffull - 64) {
    set_error("The grid exceeds 2^32 cells.");
    return PW_ERR_INVALID;
  }
  if ((body_triangles && !body) || (support_triangles && !supports)) {
    set_error("Mesh positions must match a non-negative triangle count.");
    return PW_ERR_INVALID;
  }
  // the raster kernel refuses a mesh with a coordinate that is not finite; the
  // host looks only where there is no device to run it
  cudaStream_t s;
  const cudaError_t made = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (made != cudaSuccess) {
    if (!finite_mesh(body, body_triangles) || (supports && !finite_mesh(supports, support_triangles))) {
      set_error("Mesh coordinates must be finite.");
      return PW_ERR_INVALID;
    }
    return cuda_status(made, "pw_voxelize");
  }
  pw_grid *g = new pw_grid();
  g->nx = nx; g->ny = ny; g->nz = nz; g->cells = cells;
  float *d_mesh = nullptr;
  int rc = PW_OK;
  uint8_t *votes[2] = {nullptr, nullptr};
  GridInfo *info = nullptr;
  Arena a;
  a.want((void **)&g->flags, cells * 4);
  a.want((void **)&g->qoff, cells * 4);
  cudaError_t e = a.alloc(&g->cell_arrays);
  float *d_sup = nullptr;
  if (e == cudaSuccess) e = tmp_alloc(&info, sizeof(GridInfo), s);
  if (e == cudaSuccess) e = tmp_alloc(&d_mesh, (body_triangles ? body_triangles : 1) * 36, s);
  if (e == cudaSuccess) e = tmp_alloc(&d_sup, (support_triangles ? support_triangles : 1) * 36, s);
  if (e != cudaSuccess) rc = cuda_status(e, "pw_voxelize");
  if (rc == PW_OK) {
    cudaMemsetAsync(info, 0, sizeof(GridInfo), s);
    if (body_triangles) cudaMemcpyAsync(d_mesh, body, (size_t)body_triangles * 36, cudaMemcpyHostToDevice, s);
    rc = vote_mesh(d_mesh, body_triangles, nx, ny, nz, 0, info, &votes[0], s);
  }
  if (rc == PW_OK && supports) {
    if (support_triangles) cudaMemcpyAsync(d_sup, supports, (size_t)support_triangles * 36, cudaMemcpyHostToDevice, s);
    rc = vote_mesh(d_sup, support_triangles, nx, ny, nz, 1, info, &votes[1], s);
  }
  uint2 *links = nullptr;
  if (rc == PW_OK) rc = finish_grid(g, votes[0], votes[1], floor_on, info, link_fractions ? &links : nullptr, s);
  if (rc == PW_OK && link_fractions && g->nfrac)
    rc = measure_links(g, d_mesh, body_triangles, d_sup, support_triangles, supports != nullptr, links, info, s);
  tmp_free(links, s);
  tmp_free(d_mesh, s);
  tmp_free(d_sup, s);
  tmp_free(votes[0], s);
  tmp_free(votes[1], s);
  tmp_free(info, s);
  e = cudaStreamSynchronize(s);
  if (rc == PW_OK && e != cudaSuccess) rc = cuda_status(e, "pw_voxelize");
  cudaStreamDestroy(s);
  if (rc != PW_OK) { delete g; return rc; }
  *out = g;
  return PW_OK;
}

int pw_grid_from_host(uint32_t nx, uint32_t ny, uint32_t nz, const uint32_t *geometry,
                      size_t geometry_len, const uint32_t *boundary, size_t nboundary, pw_grid **out) {
  if (!out) { set_error("out is NULL"); return PW_ERR_INVALID; }
  *out = nullptr;
  if (nx < 1 || ny < 1 || nz < 1) { set_error("Grid dimensions must be positive safe integers."); return PW_ERR_INVALID; }
  size_t cells = (size_t)nx * ny * nz;
  if (cells > 0xffffffffull - 64) { set_error("The grid exceeds 2^32 cells."); return PW_ERR_INVALID; }
  if (!geometry || geometry_len < 2 * cells) {
    set_error("Geometry must match the solver layout and contain flags and q offsets.");
    return PW_ERR_INVALID;
  }
  // q offsets and fraction count (geometry-contract.ts:7-18,50-65)
  size_t fractions = 0;
  for (size_t c = 0; c < cells; c++) {
    uint32_t flag = geometry[c], kind = flag & 7u;
    if (kind > pw::EQ) { set_error("Unknown geometry cell kind at cell %zu.", c); return PW_ERR_INVALID; }
    uint32_t off = geometry[cells + c];
    if (off == PW_NO_Q) continue;
    uint32_t mask = kind == pw::FLUID ? (flag & ~7u) : 0u;
    if (mask == 0 || off != fractions) { set_error("Invalid geometry q offset at cell %zu.", c); return PW_ERR_INVALID; }
    fractions += (size_t)__builtin_popcount(mask >> 4);
  }
  if (geometry_len != 2 * cells + fractions) {
    set_error("Geometry length must match its cell planes and packed wall-link fractions.");
    return PW_ERR_INVALID;
  }
  for (size_t k = 0; k < nboundary; k++) {
    uint32_t c = boundary[k];
    if (c >= cells || (geometry[c] & 7u) != pw::FLUID || (geometry[c] >> 4) == 0) {
      set_error("Boundary cells must index fluid cells with wall links.");
      return PW_ERR_INVALID;
    }
  }
  cudaStream_t s;
  PW_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  pw_grid *g = new pw_grid();
  g->nx = nx; g->ny = ny; g->nz = nz; g->cells = cells;
  unsigned long long *bad = nullptr;
  unsigned long long bad_h = ~0ull;
  Arena cell_arrays, link_arrays;
  cell_arrays.want((void **)&g->flags, cells * 4);
  cell_arrays.want((void **)&g->qoff, cells * 4);
  link_arrays.want((void **)&g->fractions, fractions * 4);
  link_arrays.want((void **)&g->boundary, nboundary * 4);
  cudaError_t e = cell_arrays.alloc(&g->cell_arrays);
  if (e == cudaSuccess) e = link_arrays.alloc(&g->link_arrays);
  if (e == cudaSuccess) e = cudaMalloc(&bad, 8);
  if (e == cudaSuccess) e = cudaMemcpyAsync(g->flags, geometry, cells * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(g->qoff, geometry + cells, cells * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && fractions)
    e = cudaMemcpyAsync(g->fractions, geometry + 2 * cells, fractions * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && nboundary) e = cudaMemcpyAsync(g->boundary, boundary, nboundary * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(bad, &bad_h, 8, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    validate_kernel<<<nblk(cells), 256, 0, s>>>(g->flags, nx, ny, nz, bad);
    e = cudaMemcpyAsync(&bad_h, bad, 8, cudaMemcpyDeviceToHost, s);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(bad);
  cudaStreamDestroy(s);
  if (e != cudaSuccess) { delete g; return cuda_status(e, "pw_grid_from_host"); }
  if (bad_h != ~0ull) {
    delete g;
    set_error("Inconsistent wall mask at cell %llu.", bad_h);
    return PW_ERR_INVALID;
  }
  g->nfrac = fractions;
  g->nboundary = nboundary;
  // statistics as countCells would report them (voxelize.ts:137-154)
  uint32_t solid = 0, frontal = 0, blocked = 0;
  std::vector<uint8_t> bp((size_t)ny * nz, 0), wp((size_t)ny * nz, 0);
  for (size_t c = 0; c < cells; c++) {
    uint32_t t = geometry[c] & 7u;
    if (t == pw::SOLID) { solid++; bp[c / nx] = 1; }
    if (t == pw::SOLID || t == pw::SUPPORT) wp[c / nx] = 1;
  }
  for (size_t k = 0; k < bp.size(); k++) { frontal += bp[k]; blocked += wp[k]; }
  pw_grid_stats &st = g->stats;
  st.nx = nx; st.ny = ny; st.nz = nz;
  st.solid_cells = solid; st.frontal_cells = frontal;
  st.blockage = (double)blocked / ((double)ny * nz);
  st.watertight = 1; st.missed_links = 0;
  st.geometry_len = geometry_len; st.boundary_cells = nboundary;
  *out = g;
  return PW_OK;
}

int pw_grid_stats_get(const pw_grid *grid, pw_grid_stats *out) {
  if (!grid || !out) { set_error("NULL argument"); return PW_ERR_INVALID; }
  *out = grid->stats;
  return PW_OK;
}

int pw_grid_read_geometry(const pw_grid *g, uint32_t *out, size_t capacity) {
  if (!g || !out) { set_error("NULL argument"); return PW_ERR_INVALID; }
  if (capacity < 2 * g->cells + g->nfrac) { set_error("geometry buffer too small"); return PW_ERR_INVALID; }
  PW_TRY(cudaMemcpy(out, g->flags, g->cells * 4, cudaMemcpyDeviceToHost));
  PW_TRY(cudaMemcpy(out + g->cells, g->qoff, g->cells * 4, cudaMemcpyDeviceToHost));
  if (g->nfrac) PW_TRY(cudaMemcpy(out + 2 * g->cells, g->fractions, g->nfrac * 4, cudaMemcpyDeviceToHost));
  return PW_OK;
}

int pw_grid_read_boundary(const pw_grid *g, uint32_t *out, size_t capacity) {
  if (!g || (!out && g->nboundary)) { set_error("NULL argument"); return PW_ERR_INVALID; }
  if (capacity < g->nboundary) { set_error("boundary buffer too small"); return PW_ERR_INVALID; }
  if (g->nboundary) PW_TRY(cudaMemcpy(out, g->boundary, g->nboundary * 4, cudaMemcpyDeviceToHost));
  return PW_OK;
}

void pw_grid_destroy(pw_grid *grid) { delete grid; }

}  // extern "C"
