// spatial.cu -- SpatialHash (blobs/src/spatial.rs) on the device: a point set
// with ids and radii, bucketed by integer cell, and SpatialHash::query as a
// batched radius query.
//
// The reference keys an unbounded HashMap by the cell (i32, i32) =
// ((x / cs).floor() as i32, (y / cs).floor() as i32) (spatial.rs:57-62) and a
// query visits the 3x3 cells around the query point's cell, keeping every
// point with |p - q|^2 <= (query_radius + radius)^2 (spatial.rs:155-195) --
// points further than one cell away are never seen, whatever the radius.
// Here the cells are hashed into a power-of-two table of buckets (>= 2 per
// point), points are counting-sorted by bucket, and a query walks the nine
// buckets of its neighbour cells, keeping only points whose own cell is that
// neighbour cell: buckets shared by several cells cost time, never results.
// Results of one query are returned in ascending id (the reference's order is
// its HashMap's iteration order, which is unspecified).
//
// A query is a chain of dependent loads -- bucket bounds, then the points --
// with little arithmetic, so what bounds it is how many are in flight: nine
// lanes of a group of 16 take a neighbour cell each, and the points lie in
// bucket order with their cells and ids, so that a bucket is one contiguous
// read.  (One thread walking nine buckets of indices into the points' arrays
// took 32 us to count and 59 us to write 25k queries' results.)
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "blobs_gpu.h"
#include "device.cuh"
#include "kernels.h"
#include "world.h"

using namespace blobs;

namespace {

__device__ __forceinline__ uint32_t cell_hash(int32_t cx, int32_t cy) {
  // two odd multipliers and a final avalanche (a 32-bit integer mix)
  uint32_t h = (uint32_t)cx * 0x9E3779B1u ^ ((uint32_t)cy * 0x85EBCA77u + 0x165667B1u);
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  h ^= h >> 15;
  return h;
}

struct HashDev {
  uint32_t n, mask;  // points, buckets - 1
  float cs;
  const float2* xy;
  const float* radius;
  const unsigned long long* ids;
  uint32_t* bucket;
  uint32_t* rank;
  uint32_t* count;   // per bucket, zero between builds
  uint32_t* start;   // per bucket + 1
  float4* point;     // bucket order: (x, y, radius, -)
  int2* cell;        // and the cells
  unsigned long long* id;  // and the ids
};

__global__ void __launch_bounds__(256) k_sh_keys(HashDev h) {
  pdl_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= h.n) return;
  const float2 p = h.xy[i];
  const uint32_t b = cell_hash(cell_coord(p.x, h.cs), cell_coord(p.y, h.cs)) & h.mask;
  h.bucket[i] = b;
  h.rank[i] = atomicAdd(h.count + b, 1u);
}

__global__ void __launch_bounds__(256) k_sh_scatter(HashDev h, uint32_t* status) {
  pdl_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= h.n) return;
  const uint32_t s = h.start[h.bucket[i]] + h.rank[i];
  if (s >= h.n) {
    atomicOr(status, ST_BAD_INDEX);
    return;
  }
  const float2 p = h.xy[i];
  h.point[s] = make_float4(p.x, p.y, h.radius[i], 0.0f);
  h.cell[s] = make_int2(cell_coord(p.x, h.cs), cell_coord(p.y, h.cs));
  h.id[s] = h.ids[i];
}

// In-place heap sort of a[0..n) (ascending).
__device__ void heap_sort(unsigned long long* a, uint32_t n) {
  auto sift = [&](uint32_t root, uint32_t end) {
    while (true) {
      uint32_t child = 2u * root + 1u;
      if (child >= end) return;
      if (child + 1u < end && a[child] < a[child + 1u]) ++child;
      if (!(a[root] < a[child])) return;
      const unsigned long long t = a[root];
      a[root] = a[child];
      a[child] = t;
      root = child;
    }
  };
  if (n < 2u) return;
  for (uint32_t k = n / 2u; k-- > 0u;) sift(k, n);
  for (uint32_t end = n - 1u; end > 0u; --end) {
    const unsigned long long t = a[0];
    a[0] = a[end];
    a[end] = t;
    sift(0u, end);
  }
}

constexpr uint32_t SH_LANES = 16;   // lanes of a query: one for each of its nine cells
constexpr uint32_t SH_RANKED = 64;  // results up to this many are ranked against each other, more heap-sorted

// WRITE = false: count the matches into qcount; WRITE = true: the matches'
// ids ascending from qstart[q] on in `out` (`tmp`: as much scratch, or NULL).
template <bool WRITE>
__global__ void __launch_bounds__(256) k_sh_query(HashDev h, uint32_t nq, const float2* qxy,
                                                  const float* qr, uint32_t* qcount,
                                                  const uint32_t* qstart, unsigned long long* tmp,
                                                  unsigned long long* out, unsigned long long cap) {
  pdl_enter();
  const uint32_t lane = threadIdx.x & (SH_LANES - 1u);
  const uint32_t group = 0xffffu << (threadIdx.x & 16u);  // this query's lanes of the warp
  const uint32_t q = blockIdx.x * (256u / SH_LANES) + threadIdx.x / SH_LANES;
  if (q >= nq) return;
  const float2 x = qxy[q];
  const float r = qr[q];
  // spatial.rs:139-153: the 3x3 neighbour cells (i32 arithmetic, wrapping)
  const int32_t nx = (int32_t)((uint32_t)cell_coord(x.x, h.cs) + lane / 3u - 1u);
  const int32_t ny = (int32_t)((uint32_t)cell_coord(x.y, h.cs) + lane % 3u - 1u);
  uint32_t s0 = 0, s1 = 0;
  if (lane < 9u) {
    const uint32_t b = cell_hash(nx, ny) & h.mask;
    s0 = h.start[b];
    s1 = h.start[b + 1u];
  }
  auto match = [&](uint32_t s) {
    const float4 p = h.point[s];
    const int2 c = h.cell[s];
    const float dist = r + p.z;
    const float ex = p.x - x.x, ey = p.y - x.y;
    return c.x == nx && c.y == ny && (ex * ex) + (ey * ey) <= dist * dist;
  };
  uint32_t k = 0;
  for (uint32_t s = s0; s < s1; ++s) k += match(s) ? 1u : 0u;
  uint32_t incl = k;
#pragma unroll
  for (int o = 1; o < (int)SH_LANES; o <<= 1) {
    const uint32_t y = __shfl_up_sync(group, incl, o, SH_LANES);
    if (lane >= (uint32_t)o) incl += y;
  }
  const uint32_t total = __shfl_sync(group, incl, SH_LANES - 1, SH_LANES);
  if (!WRITE) {
    if (lane == 0) qcount[q] = total;
    return;
  }
  const unsigned long long base = qstart[q];
  if (base + total > cap) return;
  const bool ranked = tmp && total <= SH_RANKED;
  unsigned long long* const to = (ranked ? tmp : out) + base;
  uint32_t at = incl - k;
  for (uint32_t s = s0; s < s1 && at < incl; ++s)
    if (match(s)) to[at++] = h.id[s];
  __syncwarp(group);
  if (ranked) {
    // (ids are unique; equal ones would keep their places)
    for (uint32_t e = lane; e < total; e += SH_LANES) {
      const unsigned long long id = to[e];
      uint32_t rank = 0;
      for (uint32_t f = 0; f < total; ++f) rank += to[f] < id || (to[f] == id && f < e) ? 1u : 0u;
      out[base + rank] = id;
    }
  } else if (lane == 0) {
    heap_sort(to, total);
  }
}

// The queries' starts as the 64-bit offsets that are handed out; the flag: a
// prefix wrapped (more than 2^32 - 1 results).
__global__ void __launch_bounds__(256) k_sh_offsets(const uint32_t* start, uint32_t n,
                                                    unsigned long long* offsets) {
  pdl_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = start[i];
  offsets[i] = s;
  if (i && s < start[i - 1u]) atomicOr(offsets + n, 1ull);
}

inline uint32_t nblk(uint64_t n) { return (uint32_t)((n + 255u) / 256u); }

// The cell scan of kernels.cu over an arbitrary count array:
// start[k] = sum(count[0..k)), start[n] = total, count zeroed.
void scan_counts(uint32_t* count, uint32_t* start, uint32_t n, uint32_t* tile_sums, uint32_t* sub_bins,
                 cudaStream_t st) {
  WorldDev d{};
  d.cell_count = count;
  d.cell_start = start;
  d.n_cells = n;
  d.n_tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  d.tile_sums = tile_sums;
  d.contacts_sub = sub_bins;
  d.defer_sub = sub_bins;
  launch_scan(d, st, true);
}

}  // namespace

struct blobs_spatial_hash {
  float cs = 1.0f;
  int device = 0;
  cudaStream_t stream = nullptr;
  uint32_t n = 0, n_buckets = 0;
  // points: ids, xy, radius, bucket, rank, and in bucket order point, cell, id;
  // buckets: count, start; scan scratch
  void* pts = nullptr;
  size_t pts_bytes = 0;
  unsigned long long *ids = nullptr, *id = nullptr;
  float2* xy = nullptr;
  float* radius = nullptr;
  float4* point = nullptr;
  int2* cell = nullptr;
  uint32_t *bucket = nullptr, *rank = nullptr, *count = nullptr, *start = nullptr;
  uint32_t *tile_sums = nullptr, *sub_bins = nullptr, *status = nullptr;
  // queries
  void* qmem = nullptr;
  size_t qmem_bytes = 0;
  void* omem = nullptr;
  size_t omem_bytes = 0;

  HashDev dev() const {
    HashDev h;
    h.n = n;
    h.mask = n_buckets ? n_buckets - 1u : 0u;
    h.cs = cs;
    h.xy = xy;
    h.radius = radius;
    h.ids = ids;
    h.bucket = bucket;
    h.rank = rank;
    h.count = count;
    h.start = start;
    h.point = point;
    h.cell = cell;
    h.id = id;
    return h;
  }
  ~blobs_spatial_hash() {
    cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);
    if (pts) cudaFree(pts);
    if (qmem) cudaFree(qmem);
    if (omem) cudaFree(omem);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

struct Carve {
  size_t off = 0;
  char* base = nullptr;
  template <class T> T* take(size_t count) {
    const size_t at = (off + 255) & ~(size_t)255;
    off = at + (count ? count * sizeof(T) : 1);
    return base ? reinterpret_cast<T*>(base + at) : nullptr;
  }
};

// (Re)allocates `mem` to hold `bytes` when it is smaller.
cudaError_t ensure(void** mem, size_t* have, size_t bytes) {
  if (*have >= bytes && *mem) return cudaSuccess;
  if (*mem) cudaFree(*mem);
  *mem = nullptr;
  *have = 0;
  cudaError_t e = cudaMalloc(mem, bytes);
  if (e == cudaSuccess) *have = bytes;
  return e;
}

}  // namespace

extern "C" {

int blobs_spatial_hash_create(float cell_size, int32_t device, blobs_spatial_hash** out) {
  if (!out) return BLOBS_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (!(cell_size > 0.0f) || !std::isfinite(cell_size)) return BLOBS_ERR_INVALID_ARGUMENT;
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) {
    cudaGetLastError();
    return BLOBS_ERR_NO_DEVICE;
  }
  if (device < 0 || device >= nd) return BLOBS_ERR_INVALID_ARGUMENT;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  blobs_spatial_hash* h = new blobs_spatial_hash();
  h->cs = cell_size;
  h->device = device;
  e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete h;
    return blobs_map_cuda(e);
  }
  *out = h;
  return BLOBS_OK;
}

int blobs_spatial_hash_destroy(blobs_spatial_hash* h) {
  if (!h) return BLOBS_ERR_INVALID_HANDLE;
  delete h;
  return BLOBS_OK;
}

int blobs_spatial_hash_set_points(blobs_spatial_hash* h, uint64_t n, const uint64_t* ids, const float* xy,
                                  const float* radius) {
  if (!h) return BLOBS_ERR_INVALID_HANDLE;
  if (n && (!ids || !xy || !radius)) return BLOBS_ERR_INVALID_ARGUMENT;
  if (n > 0x3fffffffull) return BLOBS_ERR_INVALID_ARGUMENT;
  cudaError_t e = cudaSetDevice(h->device);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  cudaStream_t st = h->stream;
  uint32_t nb = 1024;
  while (nb < 2 * n) nb <<= 1;
  const uint32_t n_tiles = (nb + SCAN_TILE - 1) / SCAN_TILE;
  auto lay = [&](Carve& c) {
    h->ids = c.take<unsigned long long>(n);
    h->xy = c.take<float2>(n);
    h->radius = c.take<float>(n);
    h->point = c.take<float4>(n);
    h->cell = c.take<int2>(n);
    h->id = c.take<unsigned long long>(n);
    h->bucket = c.take<uint32_t>(n);
    h->rank = c.take<uint32_t>(n);
    h->count = c.take<uint32_t>(nb);
    h->start = c.take<uint32_t>(nb + 1);
    h->tile_sums = c.take<uint32_t>(n_tiles);
    h->sub_bins = c.take<uint32_t>(COUNTER_BINS);
    h->status = c.take<uint32_t>(1);
  };
  Carve sizer;
  lay(sizer);
  e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = ensure(&h->pts, &h->pts_bytes, sizer.off + 256);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  Carve c;
  c.base = static_cast<char*>(h->pts);
  lay(c);
  h->n = (uint32_t)n;
  h->n_buckets = nb;
  if (n) {
    e = cudaMemcpyAsync(h->ids, ids, 8 * n, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h->xy, xy, 8 * n, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h->radius, radius, 4 * n, cudaMemcpyHostToDevice, st);
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(h->count, 0, 4 * (size_t)nb, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(h->status, 0, 4, st);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  const HashDev d = h->dev();
  if (n) launch_pdl(k_sh_keys, nblk(n), 256, st, true, d);
  scan_counts(h->count, h->start, nb, h->tile_sums, h->sub_bins, st);
  if (n) launch_pdl(k_sh_scatter, nblk(n), 256, st, true, d, h->status);
  uint32_t status = 0;
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&status, h->status, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  return status ? BLOBS_ERR_INVALID_ARGUMENT : BLOBS_OK;
}

int blobs_spatial_hash_query(blobs_spatial_hash* h, uint64_t nq, const float* qxy, const float* qradius,
                             uint64_t* offsets, uint64_t* ids, uint64_t cap, uint64_t* total) {
  if (!h) return BLOBS_ERR_INVALID_HANDLE;
  if (!total || !offsets || (nq && (!qxy || !qradius)) || (cap && !ids)) return BLOBS_ERR_INVALID_ARGUMENT;
  if (nq > 0x3fffffffull) return BLOBS_ERR_INVALID_ARGUMENT;
  *total = 0;
  offsets[0] = 0;
  if (!nq) return BLOBS_OK;
  if (!h->pts) return BLOBS_ERR_STATE;
  cudaError_t e = cudaSetDevice(h->device);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  cudaStream_t st = h->stream;
  const uint32_t n_tiles = (uint32_t)((nq + SCAN_TILE - 1) / SCAN_TILE);
  float2* dq = nullptr;
  float* dr = nullptr;
  uint32_t *qcount = nullptr, *qstart = nullptr, *tiles = nullptr, *bins = nullptr;
  unsigned long long* doff = nullptr;
  auto lay = [&](Carve& c) {
    dq = c.take<float2>(nq);
    dr = c.take<float>(nq);
    qcount = c.take<uint32_t>(nq);
    qstart = c.take<uint32_t>(nq + 1);
    tiles = c.take<uint32_t>(n_tiles);
    bins = c.take<uint32_t>(COUNTER_BINS);
    doff = c.take<unsigned long long>(nq + 2);  // the offsets, then the wrap flag
  };
  Carve sizer;
  lay(sizer);
  e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = ensure(&h->qmem, &h->qmem_bytes, sizer.off + 256);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  Carve c;
  c.base = static_cast<char*>(h->qmem);
  lay(c);
  e = cudaMemcpyAsync(dq, qxy, 8 * nq, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dr, qradius, 4 * nq, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(doff + nq + 1, 0, 8, st);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  const HashDev d = h->dev();
  const uint32_t n_off = (uint32_t)nq + 1u, blocks = nblk(nq * SH_LANES);
  launch_pdl(k_sh_query<false>, blocks, 256, st, true, d, (uint32_t)nq, dq, dr, qcount, nullptr, nullptr, nullptr, 0ull);
  // totals above 2^32 - 1 would wrap the u32 scan: refused below
  scan_counts(qcount, qstart, (uint32_t)nq, tiles, bins, st);
  launch_pdl(k_sh_offsets, nblk(n_off), 256, st, true, qstart, n_off, doff);
  unsigned long long wrapped = 0;
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(offsets, doff, 8 * (size_t)n_off, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&wrapped, doff + n_off, 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return blobs_map_cuda(e);
  if (wrapped) return BLOBS_ERR_OVERFLOW;  // the u32 prefix wrapped
  const uint64_t run = offsets[nq];
  *total = run;
  if (run > cap) return BLOBS_ERR_OVERFLOW;
  if (!run) return BLOBS_OK;
  e = ensure(&h->omem, &h->omem_bytes, 16 * run);
  const bool scratch = e == cudaSuccess;
  if (e == cudaErrorMemoryAllocation) {  // room for the results alone, perhaps
    cudaGetLastError();
    e = ensure(&h->omem, &h->omem_bytes, 8 * run);
  }
  if (e != cudaSuccess) return blobs_map_cuda(e);
  unsigned long long* dout = static_cast<unsigned long long*>(h->omem);
  launch_pdl(k_sh_query<true>, blocks, 256, st, true, d, (uint32_t)nq, dq, dr, nullptr, qstart,
             scratch ? dout + run : nullptr, dout, run);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(ids, dout, 8 * run, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return blobs_map_cuda(e);
}

}  // extern "C"
