// Parameters and small device helpers shared by the persistent Jacobi-PCG
// kernels (kernels_pcg.cu, kernels_pcg_resident.cu).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "ffg_internal.h"

namespace ffg {

constexpr int kResultDoubles = 16;
// What a solve reports: its statistics and behind them the control word
constexpr size_t kStateBytes = kResultDoubles * sizeof(double) + 2 * sizeof(int);
constexpr int kMinWindow = 256;  // iterations before a plateau forces a reliable update
constexpr unsigned long long kBarrierLimitNs = 4000000000ull;  // 4 s per barrier wait

struct PcgParams {
  int64_t n;
  const int64_t *soff;
  const int16_t *dcol;
  const int *col;
  const float *v32;
  const __half *v16;  // FFG_PRECISION_MIXED16: FP16 operator, row r scaled by rs[r]
  const float *rs;
  const double *v64;
  const float *d32;
  const double *d64;
  const int *cta_slice;
  const int *wslice, *woff;  // per-warp slice lists of the cooperative grid
  const double *b;
  double *x;
  double *r64;
  float *rf, *zf, *pf, *qf;  // mixed mode: r, z = D^-1 r, p, q = A p
  float *xf;                 // mixed mode: increment of x since it was last folded in
  float2 *zpf0, *zpf1;       // mixed mode after a switch to direct A p: (z, p) pairs
  double *rd, *qd;
  double2 *zpd0, *zpd1;
  // partial sums [2][2][grid] and the verdicts on the limit [2], or messages
  // (pcg_message_bytes)
  double *partial;
  unsigned int *bar;
  int *control;     // [0] error status
  double *result;   // kResultDoubles
  int precision, relative, max_it, max_updates, guard;
  double tol, delta;
  unsigned long long limit_ns;
  // CTAs that solve this system: blockIdx.x - cta0 in [0, ncta).  With one
  // CTA the system's slices are [0, n_slices) and barriers are CTA barriers.
  int cta0, ncta, n_slices;
  int staged;  // launched with kStageSmem bytes of dynamic shared memory
  // cluster solves: slice cuts for 8 CTAs (9), then for 16 (17), and the
  // largest count of slices of a CTA under each; share_slices the one in use
  const int *cluster_slice;
  int cluster_share[2], share_slices;
  int part_bytes;  // shared memory the parts of split slices may take
};

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned long long clock_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %clock64;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int ld_volatile_int(const int *p) {
  return *reinterpret_cast<const volatile int *>(p);
}

__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool is_finite_d(double x) { return isfinite(x); }

constexpr int kVals = 2;  // values of one reduction, at most
constexpr int kPoll = 5;            // messages a lane polls: up to 160 CTAs

struct Outcome {
  int iterations = 0, updates = 0, converged = 0, status = FFG_OK, stagnated = 0, aborted = 0;
  int restart = 0;  // the FP32 phase broke down: the FP64 loop starts again from x = 0
  double true_res = 0.0, final_res = 0.0, bnorm = 0.0;
};

// Device time of the phases seen by CTA 0 (the others are symmetric):
// SpMV work, wait at the following barrier, vector work, wait, and the
// residual-replacement phases.
struct Timing {
  unsigned long long a = 0, aw = 0, b = 0, bw = 0, u = 0;
};

// On-chip solves (kernels_pcg_resident.cu).
// CTAs of the cluster that solves a system, or 0 when it takes another kernel;
// batched: in a launch of many systems (one cluster size for all of them).
int pcg_cluster_size(const DeviceSell &A, int precision, bool batched);
// Shared memory per CTA with which the cooperative grid holds the operator on
// chip, or 0 when it does not.
size_t pcg_grid_resident(const DeviceSell &A, int precision);
// Bytes at PcgParams::partial (zero before a launch) for the messages of `ctas` CTAs.
size_t pcg_message_bytes(int ctas);
// One cluster of `cluster` CTAs per system; overlap: beside the launch of this
// kernel enqueued just before, on which it does not depend.
cudaError_t pcg_launch_cluster(int count, const PcgParams *sys, int cluster, bool batched,
                               bool overlap, cudaStream_t s);
// CTAs of the group that holds the operator in shared memory within a launch of
// several systems, or 0 when no group of up to `grid` does; max_slices: the most
// slices of one of them.
int pcg_group_shape(const DeviceSell &A, int precision, int grid, int *max_slices);
// Systems on consecutive groups of sys[i].ncta CTAs (share_slices set), at most
// kMaxResidentGroups of them, in one cooperative launch.
constexpr int kMaxResidentGroups = 16;
cudaError_t pcg_launch_resident_groups(int count, const PcgParams *sys, cudaStream_t s);
// P.ncta CTAs, cooperative.
cudaError_t pcg_launch_resident(const PcgParams &P, size_t pool_bytes, cudaStream_t s);

}  // namespace ffg
