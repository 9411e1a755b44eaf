// kernels.h -- host-side launchers of the substep kernels (kernels.cu).
#pragma once

#include "device.cuh"

namespace blobs {

// Launches a kernel that begins with pdl_enter() or pdl_enter_before_step()
// (device.cuh); early: its blocks may take their places while the kernel
// before it still drains.  The general path's chain of kernels is launched
// without: there the waiting blocks cost more than the launches (200k jointed
// bodies, four steps: 4.64 ms with, 3.64 ms without).  Such a kernel starts
// while the one before it still writes what it is going to read, so none of
// its pointers is __restrict__: that would let the compiler read through the
// non-coherent path, or move a load up across the wait.
template <class... P, class... A>
inline void launch_pdl(void (*k)(P...), uint32_t grid, uint32_t threads, cudaStream_t st, bool early, A&&... a) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, static_cast<P>(a)...);
}

void launch_keys(const WorldDev& w, bool multiworld, cudaStream_t st);
// the cell scan; returns the number of kernels it launched (early: as launch_pdl)
uint32_t launch_scan(const WorldDev& w, cudaStream_t st, bool early);
void launch_scatter_forces(const WorldDev& w, const float2* pos, bool multiworld, bool scatter, bool springs,
                           bool pending, cudaStream_t st);
uint32_t launch_contacts(const WorldDev& w, const float2* pos_in, float2* pos_out, bool multiworld, bool single,
                     bool springs, bool pending, bool fuse, float dt, float old_dt, bool do_keys, bool rot_dynamic,
                     cudaStream_t st);
void launch_joints(const WorldDev& w, float2* pos, uint32_t j0, uint32_t j1, float dt, cudaStream_t st);
void launch_joint_blocks(const WorldDev& w, float2* pos, float dt, uint32_t iterations, bool levels, cudaStream_t st);
void launch_ev_tick(const WorldDev& w, cudaStream_t st);
void launch_v_divide(float2* v, uint32_t n, float dt, cudaStream_t st);
void launch_integrate(const WorldDev& w, const float2* pos_in, float2* pos_out, bool multiworld, bool single,
                      bool springs, bool pending, float dt, float old_dt, bool do_keys, bool rot_dynamic,
                      cudaStream_t st);

void launch_emit_pairs(const WorldDev& w, bool multiworld, uint32_t mode, uint32_t* out, unsigned long long cap,
                       unsigned long long* count, cudaStream_t st);

// single-sphere path with cell-sorted storage (single.cu); mode 0: one
// uniform world, 1: one world with per-body records, 2: batched worlds, 3:
// batched uniform worlds
void launch_permute(const WorldDev& w, const SingleArgs& a, cudaStream_t st);
// with springs also the spring forces of the substep; launch_springs: those alone
void launch_scatter_cand(const WorldDev& w, const SingleArgs& a, float4* cand, cudaStream_t st);
void launch_springs(const WorldDev& w, const SingleArgs& a, cudaStream_t st);
void launch_step_single(const WorldDev& w, const SingleArgs& a, int mode, cudaStream_t st);
// the bodies the plain step deferred (after launch_step_single, same args)
void launch_step_deferred(const WorldDev& w, const SingleArgs& a, int mode, cudaStream_t st);
// whole steps of n_worlds small worlds, a cluster each; returns a cudaError_t
int launch_resident(const WorldDev& w, const ResidentArgs& r, bool uniform, uint32_t n_worlds, uint32_t shared_bytes,
                    cudaStream_t st);
void launch_keys_single(const WorldDev& w, const float4* A, int mode, cudaStream_t st);
void launch_gather_single(const WorldDev& w, const float4* A, const float4* B, const float2* V, float2* pos,
                          float2* pos_old, float2* vel, float2* snap, float v_div, cudaStream_t st);
void launch_write_single(const WorldDev& w, float4* A, float4* B, float2* V, const float2* pos,
                         const float2* pos_old, const float2* vel, const float2* snap, cudaStream_t st);

// a range of collision events put into the reference's order (events.cu)
struct EventSort {
  const uint4* rec;        // (substep sequence, a, b, 0), ascending substep
  const float4* vel;
  uint32_t n;              // events of the range
  uint32_t seq0, n_seq;    // its substeps [seq0, seq0 + n_seq), modulo 2^32
  uint32_t n_cols;
  uint32_t n_buckets;      // n_seq * n_cols
  uint32_t* count;         // n_buckets
  uint32_t* start;         // n_buckets + 1
  uint32_t* rank;          // n
  uint2* member;           // n
  uint32_t* out_a;         // n each
  uint32_t* out_b;
  float2* out_va;
  float2* out_vb;
  uint32_t* status;
};
void launch_ev_sort(const EventSort& s, uint32_t* tile_sums, cudaStream_t st);
// off[k] = index of the first event of substep seq0 + min(k * stride, n_seq)
void launch_ev_bounds(const uint4* rec, uint32_t n, uint32_t seq0, uint32_t n_seq, uint32_t stride, uint32_t* off,
                      uint32_t n_off, cudaStream_t st);

// adjoint of the single-sphere substep (adjoint.cu)
struct AdjointSubstep {
  // recorded state at the start of the substep (t) and after it (t + 1), arena order
  const float2* p_t;
  const float2* s_t;
  const float2* v_t;
  const float2* s_t1;
  const uint32_t* rec_list;  // contacts of each body in the substep, as recorded (REC_CAP x n_bodies)
  const uint32_t* rec_n;     // per body: recorded contacts
  // adjoints of the state after the substep (in) and before it (out)
  const float2* lp_in;
  const float2* lpo_in;
  const float2* ls_in;
  const float2* lv_in;
  float2* lp_out;
  float2* lpo_out;
  float2* ls_out;
  float2* lv_out;
  float2* lpc;             // scratch: adjoint of the post-contact position
  float2* la;              // scratch: adjoint of the acceleration
  float2* lv0;             // gradient of the velocity requests (first substep of the rollout)
  float* lk;               // gradient of the spring stiffnesses (accumulated)
  float4* spr_terms;       // scratch: per spring, the adjoint of d (pb - pa) and of rv (va - vb)
  float dt;
  float ratio_first;       // dt / old_dt for the first dynamic body (first substep only)
  uint32_t first_substep;  // the rollout's first substep (dt / old_dt applies)
  uint32_t vreq_pending;   // velocity requests were pending at the rollout's start
};
// the body part of a substep alone
void launch_adjoint_body(const WorldDev& w, const AdjointSubstep& a, cudaStream_t st);
// the spring and gather parts of a substep whose body part is done, and the
// body part of the substep before it (NULL: there is none)
void launch_adjoint_substep(const WorldDev& w, const AdjointSubstep& a, const AdjointSubstep* before, cudaStream_t st);

}  // namespace blobs
