// events.cu -- the collision-event buffer put into the reference's order on
// the device: substep by substep, outer collider ascending, inner collider
// ascending (physics.rs:247-248).
//
// The contact kernels append a substep's events in any order, and the
// substeps one after the other, so the buffer is ordered by substep already.
// What is left is a counting sort by (substep, a) -- one bucket per collider
// and substep, through the cell scan -- and the few events of one bucket (a
// body's contacts with lower ids) ranked by b against each other.  Each
// event is read three times and written once (16 + 16 + 32 B in, 24 B out),
// and the buckets cost 16 B each: bound by launches below ~1e6 events and by
// the scattered bucket accesses above.  A radix sort of the 96-bit keys
// would pass over all events a dozen times.
// A frame of 20k spheres with ~75k events (step, drain, read): 0.50 ms; with
// the records copied out and sorted by std::sort on the host it took 5.28 ms.
#include "device.cuh"
#include "kernels.h"

namespace blobs {

// bucket of event i: (its substep - seq0) * n_cols + a; n_buckets when it
// has none in this range (never, unless the buffer is corrupt)
__device__ __forceinline__ uint32_t event_bucket(const EventSort& s, uint4 r) {
  const uint32_t rel = r.x - s.seq0;
  return rel < s.n_seq && r.y < s.n_cols ? rel * s.n_cols + r.y : s.n_buckets;
}

// first event of each substep of the batch: off[k] = lower bound of seq0 + k
__global__ void __launch_bounds__(256) k_ev_bounds(const uint4* rec, uint32_t n, uint32_t seq0,
                                                   uint32_t n_seq, uint32_t stride, uint32_t* off,
                                                   uint32_t n_off) {
  pdl_enter();
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_off) return;
  const uint32_t want = min(k * stride, n_seq);
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2u;
    if (rec[mid].x - seq0 < want) lo = mid + 1u;
    else hi = mid;
  }
  off[k] = lo;
}

__global__ void __launch_bounds__(256) k_ev_count(EventSort s) {
  pdl_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  const uint32_t k = event_bucket(s, s.rec[i]);
  if (k < s.n_buckets) s.rank[i] = atomicAdd(s.count + k, 1u);
  else atomicOr(s.status, ST_BAD_INDEX);
}

// member[slot] = (b, event) of the event at its place among the buckets
__global__ void __launch_bounds__(256) k_ev_place(EventSort s) {
  pdl_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  const uint4 r = s.rec[i];
  const uint32_t k = event_bucket(s, r);
  if (k >= s.n_buckets) return;
  const uint32_t slot = s.start[k] + s.rank[i];
  if (slot < s.n) s.member[slot] = make_uint2(r.z, i);
}

// one thread per event: its rank by b inside its bucket is its place
// (pairs are distinct; the slot breaks ties so that ranks stay a permutation)
__global__ void __launch_bounds__(256) k_ev_write(EventSort s) {
  pdl_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  const uint4 r = s.rec[i];
  const uint32_t k = event_bucket(s, r);
  if (k >= s.n_buckets) return;
  const uint32_t q0 = s.start[k], q1 = min(s.start[k + 1u], s.n), own = q0 + s.rank[i];
  uint32_t at = q0;
  for (uint32_t q = q0; q < q1; ++q) {
    const uint32_t b = s.member[q].x;
    at += (b < r.z || (b == r.z && q < own)) ? 1u : 0u;
  }
  if (at >= s.n) return;
  const float4 v = s.vel[i];
  s.out_a[at] = r.y;
  s.out_b[at] = r.z;
  s.out_va[at] = v2(v.x, v.y);
  s.out_vb[at] = v2(v.z, v.w);
}

void launch_ev_bounds(const uint4* rec, uint32_t n, uint32_t seq0, uint32_t n_seq, uint32_t stride, uint32_t* off,
                      uint32_t n_off, cudaStream_t st) {
  launch_pdl(k_ev_bounds, (n_off + 255u) / 256u, 256, st, true, rec, n, seq0, n_seq, stride, off, n_off);
}

void launch_ev_sort(const EventSort& s, uint32_t* tile_sums, cudaStream_t st) {
  if (!s.n) return;
  const uint32_t g = (s.n + 255u) / 256u;
  cudaMemsetAsync(s.count, 0, sizeof(uint32_t) * (size_t)s.n_buckets, st);
  launch_pdl(k_ev_count, g, 256, st, true, s);
  WorldDev d{};  // the cell scan over the buckets
  d.cell_count = s.count;
  d.cell_start = s.start;
  d.n_cells = s.n_buckets;
  d.n_tiles = (s.n_buckets + SCAN_TILE - 1) / SCAN_TILE;
  d.tile_sums = tile_sums;
  launch_scan(d, st, true);
  launch_pdl(k_ev_place, g, 256, st, true, s);
  launch_pdl(k_ev_write, g, 256, st, true, s);
}

}  // namespace blobs
