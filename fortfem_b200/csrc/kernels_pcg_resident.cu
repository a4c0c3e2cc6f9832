// On-chip Jacobi-PCG (sm_100a): the solves of kernels_pcg.cu for systems whose
// operator fits the shared memory of the CTAs that solve it.
//
// The values and column indices of a CTA's slices are copied into its shared
// memory once per solve, and the iteration vectors of its rows (r, p, q, D^-1,
// the step of x) live there too; an iteration moves only the published
// vector (the operand of A) and the partial sums of the dot products between
// CTAs.  What bounds it is latency: two reductions an iteration.  Per
// iteration and solve, measured on a B200 against the kernels it replaces:
// P1, 3,969 rows, 2.5 us (14 us with 148 CTAs and grid barriers); P1, 85,800
// rows, 7.5 us (13.6); P2, 71,955 rows, 10.5 us (20.0); a batch of 12 systems of
// 961 to 21,025 rows 3.5 ms (41 ms with one CTA a system).
//
// * pcg_cluster_kernel: a thread-block cluster per system.  Every CTA holds a
//   replica of the published vector, and the owners copy the slices that
//   another CTA reads into its replica through distributed shared memory, so
//   the SpMV gathers from its own shared memory; a reduction is one round of
//   st.async messages counted by mbarriers.  Clusters wait on nothing outside
//   themselves, so launches of this kernel may overlap.
// * pcg_resident_kernel: one cooperative grid per system.  The published vector
//   is in global memory (L2); a reduction is an all-to-all of messages, one per
//   CTA, polled by every CTA: the message carries the partial sums and is its
//   own arrival flag.
//
// Slices that do not fit stay in global memory and are read from L2.  The
// recurrences, stopping rules and fallbacks are those of kernels_pcg.cu; the
// FP64 loop and the direct form of the mixed loop publish p itself (one more
// sync, without sums) where kernels_pcg.cu gathers (z, p) pairs.  All sums are
// taken in a fixed order that depends on the system and its CTA count alone.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <mutex>

#include "cluster_phase.h"
#include "pcg_common.cuh"

namespace ffg {

namespace {

constexpr int kGridThreads = 512;
constexpr int kMaxCluster = 16;
constexpr int kBatch = 8;          // columns of a row in flight
constexpr int kPoolMax = 225 * 1024;
constexpr unsigned long long kLandNs = 1000000;  // far above a message's time of about 1 us

// Before the grid's first poll of a sync: the polls of 148 CTAs hit the same few
// L2 lines and slow the messages and the fences they wait for (P1, 85,800
// rows: 9.4 us an iteration without naps, 7.8 with these; between polls a nap
// gained nothing).
constexpr unsigned kNapSums = 200, kNapData = 700;  // ns


// A slice of this CTA: where it starts in the operator, in the CTA's
// shared-memory copy (-1: not copied), and its length in columns.
struct SliceEnt {
  int64_t goff;
  int off, len;
  int part0;          // first scratch row of its parts, when it has several
  int parts, cols;     // column parts it is split into, columns of a part
};

struct ResShared {
  double red[kVals][16], res[kVals];
  double slot[2][kVals][kMaxCluster];
  // the wall limit; past_limit, deadline: the first CTA's first thread's own
  unsigned long long deadline;
  int past_limit;  // its last look, which it takes while it waits in a phase
  int late;        // grid: the first CTA's verdict
  unsigned long long mbar[2];
  unsigned long long mbar_all[2];  // the cluster's barrier
  int ok, items, rows;
  int need;               // slices that arrive in an exchange
  int2 send[kMaxCluster]; // this CTA's slices [x, y) that CTA k reads
};
__shared__ PcgParams gP;   // the system of this CTA
__shared__ ResShared gSh;

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__device__ __forceinline__ unsigned mapa(unsigned addr, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// Sums of v[0..NV) over the CTA, for warp 0: lanes 0-15 get the first,
// lanes 16-31 the second.  Two values share the butterfly after one exchange.
template <int NV, int NT>
__device__ __forceinline__ double block_sums(const double (&v)[kVals]) {
  static_assert(NT <= 512, "16 warps");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4;
  double x;
  if (NV == 2) {
    x = half ? v[1] : v[0];
    x += __shfl_xor_sync(0xffffffffu, half ? v[0] : v[1], 16);
  } else {
    x = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if ((lane & 15) == 0 && half < NV) gSh.red[half][warp] = x;
  __syncthreads();
  if (warp == 0) {
    x = (half < NV && (lane & 15) < NT / 32) ? gSh.red[half][lane & 15] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  }
  return x;
}

// What the first CTA sends for its second sum once the wall limit has passed: a
// signalling NaN, which no arithmetic
// returns.  A message or a register of its own for the verdict cost the grid
// 1.5 us an iteration in spilled registers.
constexpr long long kLate = 0x7ff4000000000001ll;

// ------------------------------------------------------------ synchronisation
// sums<NV>(v, out): the sums of the threads' v[0..NV) over all CTAs of the
// system, the same bits in every thread.  Every load whose value went into a
// sum has completed before any CTA goes on, but no other memory is ordered.
// reduce<NV>(v, out) also releases and acquires all earlier writes (NV = 0:
// the barrier alone).  False: give up.  With a second sum
// comes the first CTA's verdict on the wall limit: late(), to be read before the
// next phase.

// Sums travel by st.async into every CTA's slots, each counting on the
// receiver's mbarrier, which the receiver alone waits for (with its own
// bound): 1300 cycles for two sums over 8 CTAs of 512 threads, against 1600
// with plain remote stores and barrier.cluster (16 CTAs: 1450 against 2050).
// Every phase waits for a message of every CTA, sums or not (cluster_phase.h):
// the two slot sets and mbarriers are safe to reuse only then.
// Every wait is bounded, so every CTA comes to rendezvous() at the kernel's end,
// also after it or another one gave up: barrier.cluster has no bound, and a
// barrier of the solve that used it would pair with the last one of a CTA that
// gave up, let that CTA leave, and have later sums sent to its shared memory.
template <int NT>
struct ClusterSync {
  int rank, n;
  unsigned phase, turn;  // turn: barriers so far

  // At the kernel's start and end alone.
  __device__ __forceinline__ void rendezvous() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }

  // Warp 0 waits, for kBarrierLimitNs, for the mbarrier's phase of this parity.
  __device__ __forceinline__ void wait(unsigned mbar, unsigned parity) {
    unsigned long long t0 = 0;
    for (unsigned spin = 1;; ++spin) {
      unsigned done;
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
          " selp.u32 %0, 1, 0, p;\n}"
          : "=r"(done)
          : "r"(mbar), "r"(parity)
          : "memory");
      if (__all_sync(0xffffffffu, done)) return;
      if ((spin & 255u) == 0) {
        if (t0 == 0) t0 = globaltimer();
        if (__any_sync(0xffffffffu, globaltimer() - t0 > kBarrierLimitNs)) {
          if ((threadIdx.x & 31) == 0) gSh.ok = 0;
          return;
        }
      }
    }
  }

  // All writes of the cluster before it are visible after it.  Two mbarriers in
  // turn: a CTA arrives again at one of them only after the barrier between,
  // for which every CTA has finished its wait here.
  __device__ __forceinline__ bool barrier() {
    const int lane = threadIdx.x & 31;
    const unsigned mbar = smem_addr(&gSh.mbar_all[++turn & 1u]);
    __syncthreads();
    if (threadIdx.x < 32) {
      if (lane < n)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                         mapa(mbar, lane))
                     : "memory");
      __syncwarp();
      wait(mbar, ((turn - 1) >> 1) & 1u);
    }
    __syncthreads();
    return gSh.ok != 0;
  }

  // sums<NV>, and with `base` the exchange of a replicated vector of
  // `slice_bytes` a slice: the slices gSh.send[k] go to the same place of CTA
  // k, by bulk copies from this CTA's shared memory.
  template <int NV>
  __device__ __forceinline__ bool sums(const double (&v)[kVals], double (&out)[kVals],
                                       const void *base = nullptr, unsigned slice_bytes = 0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4, l = lane & 15;
    const unsigned par = ++phase & 1u;
    constexpr int NM = phase_messages(NV);
    const unsigned mbar = smem_addr(&gSh.mbar[par]);
    // the rows written by ordinary stores are read by the copy engine
    if (base) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    double x = 0.0;
    if (NV > 0) x = block_sums<NV, NT>(v);
    else __syncthreads();
    if (base && warp == 1 && lane < n && lane != rank) {
      const int2 part = gSh.send[lane];
      if (part.y > part.x) {
        const unsigned src = smem_addr(base) + part.x * slice_bytes;
        asm volatile(
            "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                mapa(src, lane)),
            "r"(src), "r"((part.y - part.x) * slice_bytes), "r"(mapa(mbar, lane))
            : "memory");
      }
    }
    if (warp == 0) {
      if (NV == 2 && rank == 0 && __shfl_sync(0xffffffffu, gSh.past_limit, 0) && half)
        x = __longlong_as_double(kLate);
      if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar),
                     "r"(phase_bytes(NV, n, base ? gSh.need * slice_bytes : 0u))
                     : "memory");
      if (l < n && half < NM)
        asm volatile(
            "st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                mapa(smem_addr(&gSh.slot[par][half][rank]), l)),
            "l"(__double_as_longlong(x)), "r"(mapa(mbar, l))
            : "memory");
      __syncwarp();
      if (rank == 0 && lane == 0) gSh.past_limit = globaltimer() > gSh.deadline;
      // for everything this phase expects
      wait(mbar, ((phase - 1) >> 1) & 1u);
    }
    __syncthreads();
    if (NV > 0) {
      x = (half < NV && l < n) ? gSh.slot[par][half][l] : 0.0;
#pragma unroll
      for (int o = kMaxCluster / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
#pragma unroll
      for (int s = 0; s < NV; ++s) out[s] = __shfl_sync(0xffffffffu, x, 16 * s);
    }
    return gSh.ok != 0;
  }
  __device__ __forceinline__ bool late() const {
    return __double_as_longlong(gSh.slot[phase & 1u][1][0]) == kLate;
  }

  template <int NV>
  __device__ __forceinline__ bool reduce(const double (&v)[kVals], double (&out)[kVals]) {
    if (!barrier()) return false;
    return NV > 0 ? sums<NV>(v, out) : true;
  }
};

// A grid message: 16 bytes per value, [parity][value][CTA], a double split in
// halves that each carry the phase below them, so that every 8-byte element
// validates itself.  The polled sectors are what a sync costs beyond latency:
// with the two values of a CTA side by side, 32 bytes read by two loads, a sync
// with two sums took 4.7 us where this layout takes 3.4.
// Every CTA calls the same syncs in the same order; msg is zero before the launch.
// kGroup: instantiated once per kernel.
template <int NT, bool kGroup>
struct GridSync {
  int rank, n;
  unsigned phase;

  template <int NV>
  __device__ __forceinline__ bool sums(const double (&v)[kVals], double (&out)[kVals]) {
    return go<NV, false>(v, out);
  }
  template <int NV>
  __device__ __forceinline__ bool reduce(const double (&v)[kVals], double (&out)[kVals]) {
    return go<NV, true>(v, out);
  }

  template <int NV, bool kData>
  __device__ __forceinline__ bool go(const double (&v)[kVals], double (&out)[kVals]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NM = NV > 0 ? NV : 1;  // values a message carries
    ++phase;
    double x = 0.0;
    if (NV > 0) x = block_sums<NV, NT>(v);
    else __syncthreads();
    if (warp == 0) {
      unsigned long long *slots =
          reinterpret_cast<unsigned long long *>(gP.partial) + (size_t)(phase & 1u) * 4 * n;
      const double x1 = __shfl_sync(0xffffffffu, x, 16);
      if (lane == 0) {
        // release: the CTA's writes before the __syncthreads, then the message
        if (kData) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        unsigned long long e[4];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          unsigned long long bits = (unsigned long long)__double_as_longlong(s ? x1 : x);
          if (NV == 2 && s == 1 && rank == 0 && gSh.past_limit) bits = kLate;
          e[2 * s] = (bits << 32) | phase;
          e[2 * s + 1] = (bits & 0xffffffff00000000ull) | phase;
        }
#pragma unroll
        for (int s = 0; s < NM; ++s)
          asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(slots + 2 * (s * n + rank)),
                       "l"(e[2 * s]), "l"(e[2 * s + 1])
                       : "memory");
      }
      if (rank == 0 && lane == 0) gSh.past_limit = globaltimer() > gSh.deadline;
      __syncwarp();
      __nanosleep(kData ? kNapData : kNapSums);
      unsigned long long e[kPoll][4], t0 = 0;
      unsigned spins = 0;
      bool good = true;
      while (true) {
        bool here = true;
#pragma unroll
        for (int k = 0; k < kPoll; ++k) {
          if (lane + 32 * k < n)
#pragma unroll
            for (int s = 0; s < NM; ++s)
              asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                           : "=l"(e[k][2 * s]), "=l"(e[k][2 * s + 1])
                           : "l"(slots + 2 * (s * n + lane + 32 * k))
                           : "memory");
        }
#pragma unroll
        for (int k = 0; k < kPoll; ++k)
          if (lane + 32 * k < n)
#pragma unroll
            for (int j = 0; j < 2 * NM; ++j) here = here && (unsigned)e[k][j] == phase;
        if (__all_sync(0xffffffffu, here)) break;
        if ((++spins & 255u) == 0) {
          if (t0 == 0) t0 = globaltimer();
          const bool late = globaltimer() - t0 > kBarrierLimitNs;
          if (late && lane == 0) atomicCAS(gP.control, 0, FFG_TIMEOUT);
          if (__any_sync(0xffffffffu, late || ld_volatile_int(gP.control) != 0)) {
            good = false;
            break;
          }
        }
      }
      // acquire: what the other CTAs wrote before their messages
      if (kData) asm volatile("fence.acq_rel.gpu;" ::: "memory");
      double acc[kVals] = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < kPoll; ++k)
        if (lane + 32 * k < n) {
#pragma unroll
          for (int s = 0; s < NV; ++s)
            acc[s] += __longlong_as_double((long long)((e[k][2 * s] >> 32) |
                                                       (e[k][2 * s + 1] & 0xffffffff00000000ull)));
        }
#pragma unroll
      for (int s = 0; s < NV; ++s) acc[s] = warp_sum(acc[s]);
      if (lane == 0) {
#pragma unroll
        for (int s = 0; s < NV; ++s) gSh.res[s] = acc[s];
        // this lane's first message is the first CTA's
        if (NV == 2) gSh.late = ((e[0][2] >> 32) | (e[0][3] & 0xffffffff00000000ull)) == kLate;
        if (!good) gSh.ok = 0;
      }
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NV; ++s) out[s] = gSh.res[s];
    return gSh.ok != 0;
  }
  __device__ __forceinline__ bool late() const { return gSh.late != 0; }
};

// ------------------------------------------------------------------- a solve
// IDX: how the columns of the shared-memory copy are kept.
constexpr int kAbs16 = 0;   // uint16 column (the published vector is in shared memory)
constexpr int kRel16 = 1;   // int16 column - row
constexpr int kAbs32 = 2;   // int32 column

extern __shared__ __align__(128) unsigned char res_pool[];

// A CTA's rows: slices s0 .. s0 + nsl - 1.
struct Share {
  int s0, nsl;
  int tab_slices;  // slice table entries, the same in every CTA of a cluster
  unsigned pool_bytes, part_bytes;  // dynamic shared memory, and what parts of slices may take of it
};

template <class Sync, int IDX, int NT>
struct Solve {
  Sync S;
  unsigned char *pool;  // dynamic shared memory after the slice table
  unsigned pool_bytes;
  SliceEnt *tab;
  int nsl, s0;
  int R;                // local rows (32 nsl)
  // The SpMV's unit of work: a column part of a slice, so that long slices
  // spread over the warps (item: slice, part << 16).  The partial sums of a
  // slice with several parts go to scratch (16 bytes a row) and are added in
  // column order; a slice of one part is finished at once.
  int items, scratch_rows;
  unsigned *item;
  int tid, lane, warp;
  // laid out by setup<V>
  unsigned char *pub, *scratch, *mval, *midx, *vec;

  static constexpr int kIdxBytes = IDX == kAbs32 ? 4 : 2;

  template <typename V> __device__ __forceinline__ V *vecs(int k) { return reinterpret_cast<V *>(vec) + (size_t)k * R; }
  __device__ __forceinline__ int row_of(int li) const {
    return s0 * kSliceRows + li;
  }
  template <class F> __device__ __forceinline__ void for_rows(F f) {
    for (int li = tid; li < R; li += NT) {
      const int row = row_of(li);
      if (row < gP.n) f(li, row);
    }
  }

  // Shared-memory layout for value type V and the copy of the slices that fit.
  template <typename V>
  __device__ __forceinline__ void setup(const V *val) {
    unsigned char *at = pool, *end = pool + pool_bytes;
    auto take = [&](size_t bytes) {
      unsigned char *q = at;
      at += (bytes + 127) & ~(size_t)127;
      return q;
    };
    // first, at the same offset in every CTA of the cluster
    if (IDX == kAbs16) pub = take((size_t)gP.n_slices * kSliceRows * sizeof(V));
    unsigned char *need = IDX == kAbs16 ? take(gP.n_slices) : nullptr;
    vec = take((size_t)5 * R * sizeof(V));
    scratch = take((size_t)scratch_rows * 32 * sizeof(double2));
    const int cap = end > at ? (int)((size_t)(end - at) / ((sizeof(V) + kIdxBytes) * 32)) * 32 : 0;
    mval = at;
    midx = at + (size_t)cap * sizeof(V);
    __syncthreads();
    if (warp == 0) {
      int sum = 0;
      for (int i0 = 0; i0 < nsl; i0 += 32) {
        const int i = i0 + lane, e = i < nsl ? tab[i].len * 32 : 0;
        int x = e;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (i < nsl) tab[i].off = sum + x <= cap ? sum + x - e : -1;
        sum += __shfl_sync(0xffffffffu, x, 31);
      }
    }
    __syncthreads();
    V *sv = reinterpret_cast<V *>(mval);
    for (int i = warp; i < nsl; i += NT / 32) {
      const SliceEnt t = tab[i];
      if (t.off < 0) continue;
      const int row = row_of(32 * i + lane);
      with_columns(row, [&](auto col) {
#pragma unroll 4
        for (int j = 0; j < t.len; ++j) {
          const int64_t e = t.goff + (int64_t)j * 32 + lane;
          const int d = t.off + j * 32 + lane;
          const V a = __ldcs(val + e);
          const int c = col(e);
          sv[d] = a;
          if (IDX == kAbs32) reinterpret_cast<int *>(midx)[d] = c;
          else if (IDX == kRel16) reinterpret_cast<int16_t *>(midx)[d] = (int16_t)(c - row);
          else reinterpret_cast<uint16_t *>(midx)[d] = (uint16_t)c;
        }
      });
    }
    __syncthreads();
    if constexpr (IDX == kAbs16) exchange_plan(need);
  }

  // Which slices of every other CTA this one's columns lie in: the first and
  // last of each CTA's range, told to their owner.  A banded system (P1 in its
  // natural order) exchanges its borders only; distributed shared memory moves
  // about 10 bytes a clock and SM, so the replica of 19,321 rows took 4 us an
  // iteration where its borders take the sync alone.
  __device__ __forceinline__ void exchange_plan(unsigned char *need) {
    for (int i = tid; i < gP.n_slices; i += NT) need[i] = 0;
    if (tid == 0) gSh.need = 0;
    __syncthreads();
    for (int i = warp; i < nsl; i += NT / 32) {
      const SliceEnt t = tab[i];
      const int row = row_of(32 * i + lane);
      if (t.off >= 0) {
#pragma unroll 4
        for (int j = 0; j < t.len; ++j) need[column(row, t.off + j * 32 + lane) >> 5] = 1;
      } else {
        with_columns(row, [&](auto col) {
#pragma unroll 4
          for (int j = 0; j < t.len; ++j) need[col(t.goff + (int64_t)j * 32 + lane) >> 5] = 1;
        });
      }
    }
    __syncthreads();
    for (int c = warp; c < S.n; c += NT / 32) {
      int lo = INT_MAX, hi = 0;
      for (int i = gP.cta_slice[c] + lane; i < gP.cta_slice[c + 1]; i += 32)
        if (need[i]) {
          lo = min(lo, i);
          hi = max(hi, i + 1);
        }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if (lo > hi) lo = hi;
      if (lane == 0 && c != S.rank) {
        atomicAdd(&gSh.need, hi - lo);
        asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};" ::"r"(
                         mapa(smem_addr(&gSh.send[S.rank]), c)),
                     "r"(lo), "r"(hi)
                     : "memory");
      }
    }
    S.barrier();  // what fails here is seen by the sums that follow
  }

  template <typename V> __device__ __forceinline__ V *published() {
    if (IDX == kAbs16) return reinterpret_cast<V *>(pub);
    return sizeof(V) == 4 ? reinterpret_cast<V *>(gP.zf) : reinterpret_cast<V *>(gP.rd);
  }
  // Row `row` of the published vector, for every CTA to read after exchange().
  // A replica's rows are the source of the copies of the exchange before: a
  // phase of sums or a barrier lies between the two, after which every CTA has
  // received them.
  template <typename V> __device__ __forceinline__ void publish(int row, V v) {
    published<V>()[row] = v;
  }
  // The rows published by every CTA become visible to all, with sums<NV>.
  template <typename V, int NV>
  __device__ __forceinline__ bool exchange(const double (&v)[kVals], double (&out)[kVals]) {
    if constexpr (IDX == kAbs16) {
      return S.template sums<NV>(v, out, pub, kSliceRows * (unsigned)sizeof(V));
    } else {
      return S.template reduce<NV>(v, out);
    }
  }

  // Column of entry d of the shared-memory copy.
  __device__ __forceinline__ int column(int row, int d) const {
    if (IDX == kAbs32) return reinterpret_cast<const int *>(midx)[d];
    if (IDX == kRel16) return row + (int)reinterpret_cast<const int16_t *>(midx)[d];
    return reinterpret_cast<const uint16_t *>(midx)[d];
  }

  // Calls f with what reads the column of an operator entry from global memory
  // (one instance of f's loop per index width: a branch in the loop would end
  // the overlap of its loads).
  template <class F> __device__ __forceinline__ void with_columns(int row, F f) {
    if (IDX == kRel16 || (IDX == kAbs16 && gP.dcol)) {
      const int16_t *dcol = gP.dcol;
      f([=](int64_t e) { return row + (int)dcol[e]; });
    }
    if (IDX == kAbs32 || (IDX == kAbs16 && !gP.dcol)) {
      const int *col = gP.col;
      f([=](int64_t e) { return col[e]; });
    }
  }

  // f(j, true) for the columns j in [j0, j1), kBatch at a time so that their
  // loads are in flight together; the last batch is filled up with f(j1 - 1, false).
  template <class F> __device__ __forceinline__ void batches(int j0, int j1, F f) {
    for (; j0 + kBatch <= j1; j0 += kBatch) {
#pragma unroll
      for (int u = 0; u < kBatch; ++u) f(j0 + u, true);
    }
    if (j0 < j1) {
#pragma unroll
      for (int u = 0; u < kBatch; ++u) f(min(j0 + u, j1 - 1), j0 + u < j1);
    }
  }

  // f(slice, its entry, part, first and last column) for this warp's items.
  template <class F> __device__ __forceinline__ void for_items(F f) {
    for (int q = warp; q < items; q += NT / 32) {
      const unsigned it = item[q];
      const int i = (int)(it & 0xffffu), k = (int)(it >> 16);
      const SliceEnt t = tab[i];
      f(i, t, k, k * t.cols, min(t.len, (k + 1) * t.cols));
    }
  }

  // fin(li, row, sum over the row's entries of value * published[column]) for
  // every local row, the thread's sum of what fin returns.
  template <typename V, class F>
  __device__ __forceinline__ double spmv(const V *val, F fin) {
    const V *z = published<V>();
    const V *sv = reinterpret_cast<const V *>(mval);
    V *part = reinterpret_cast<V *>(scratch);
    double dot = 0.0;
    for_items([&](int i, const SliceEnt &t, int k, int j0, int j1) {
      const int row = row_of(32 * i + lane);
      V acc = 0;
      if (t.off >= 0) {
        batches(j0, j1, [&](int j, bool in) {
          const int d = t.off + j * 32 + lane;
          const V a = in ? sv[d] : V(0);
          acc += a * z[column(row, d)];
        });
      } else {
        with_columns(row, [&](auto col) {
          batches(j0, j1, [&](int j, bool in) {
            const int64_t e = t.goff + (int64_t)j * 32 + lane;
            const V a = in ? val[e] : V(0);  // again next iteration: kept in L2
            acc += a * z[col(e)];
          });
        });
      }
      if (t.parts > 1) part[(t.part0 + k) * 32 + lane] = acc;
      else if (row < gP.n) dot += fin(32 * i + lane, row, acc);
    });
    if (scratch_rows > 0) {
      __syncthreads();
      for_rows([&](int li, int row) {
        const SliceEnt &t = tab[li >> 5];
        if (t.parts == 1) return;
        const V *at = part + t.part0 * 32 + (li & 31);
        V acc = at[0];
        for (int k = 1; k < t.parts; ++k) acc += at[32 * k];
        dot += fin(li, row, acc);
      });
    }
    return dot;
  }

  // r64 = b - A x with the FP64 operator (x in global memory); with kP also
  // q = A p from the published p, in FP64.  Returns the thread's share of (r64, r64).
  template <bool kP>
  __device__ __forceinline__ double residual(float *q) {
    const float *p = published<float>();
    const double *x = gP.x, *v64 = gP.v64;
    double2 *part = reinterpret_cast<double2 *>(scratch);
    double dot = 0.0;
    auto fin = [&](int li, int row, double ax, double ap) {
      const double r = gP.b[row] - ax;
      gP.r64[row] = r;
      if (kP) q[li] = (float)ap;
      dot += r * r;
    };
    for_items([&](int i, const SliceEnt &t, int k, int j0, int j1) {
      const int li = 32 * i + lane, row = row_of(li);
      double ax = 0.0, ap = 0.0;
      auto add = [&](int64_t e, int c, bool in) {
        const double v = in ? __ldcs(v64 + e) : 0.0;
        ax += v * x[c];
        if (kP) ap += v * (double)p[c];
      };
      if (t.off >= 0) {
        batches(j0, j1, [&](int j, bool in) {
          add(t.goff + (int64_t)j * 32 + lane, column(row, t.off + j * 32 + lane), in);
        });
      } else {
        with_columns(row, [&](auto col) {
          batches(j0, j1, [&](int j, bool in) {
            const int64_t e = t.goff + (int64_t)j * 32 + lane;
            add(e, col(e), in);
          });
        });
      }
      if (t.parts > 1) part[(t.part0 + k) * 32 + lane] = make_double2(ax, ap);
      else if (row < gP.n) fin(li, row, ax, ap);
    });
    __syncthreads();
    if (scratch_rows > 0) {
      for_rows([&](int li, int row) {
        const SliceEnt &t = tab[li >> 5];
        if (t.parts == 1) return;
        const double2 *at = part + t.part0 * 32 + (li & 31);
        double2 a = at[0];
        for (int k = 1; k < t.parts; ++k) {
          a.x += at[32 * k].x;
          a.y += at[32 * k].y;
        }
        fin(li, row, a.x, a.y);
      });
      __syncthreads();
    }
    return dot;
  }

  __device__ __forceinline__ bool residual_norms(double (&red)[kVals]) {
    if (tid == 0) gSh.past_limit = 0;  // (b, b) is a sum, not a verdict
    double part[kVals] = {residual<false>(nullptr), 0.0};
    for_rows([&](int, int row) {
      const double bb = gP.b[row];
      part[1] += bb * bb;
    });
    return S.template sums<2>(part, red);
  }

  __device__ __forceinline__ bool barrier() {
    double none[kVals], out[kVals];
    return S.template reduce<0>(none, out);
  }

  __device__ __forceinline__ unsigned long long stamp() const {
    return (S.rank == 0 && tid == 0) ? clock_now() : 0ull;
  }

  // cg64 of kernels_pcg.cu: the reference's recurrences (or, after a stagnated
  // mixed solve, its continuation in restarted cycles).
  __device__ __forceinline__ void fp64(bool continuation, Outcome &o,
                                    Timing &tm) {
    setup<double>(gP.v64);
    double *r = vecs<double>(0), *p = vecs<double>(1), *q = vecs<double>(2), *d = vecs<double>(3),
           *x = vecs<double>(4);
    double part[kVals] = {0, 0}, red[kVals];
    unsigned long long t0, t1, t2;
    t0 = stamp();
    if (!residual_norms(red)) { o.aborted = 1; return; }
    const double bnorm = sqrt(red[1]), rnorm = sqrt(red[0]);
    o.bnorm = bnorm;
    const double target = gP.relative ? gP.tol * (continuation ? bnorm : rnorm) : gP.tol;
    double true_res = rnorm, last_true = rnorm;
    int stall = 0, cycle_its = 0, first_cycle = 0;
    int converged = rnorm <= target ? 1 : 0;
    double rz = 0.0;
    if (!converged) {
      part[0] = 0.0;
      for_rows([&](int li, int row) {
        const double rr = gP.r64[row], dd = gP.d64[row];
        r[li] = rr;
        d[li] = dd;
        p[li] = 0.0;
        x[li] = gP.x[row];
        part[0] += rr * (dd * rr);
      });
      if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
      rz = red[0];
    }
    tm.u += stamp() - t0;
    // the residual estimate, squared, against the target, squared
    double beta = 0.0, est2 = rnorm * rnorm;
    const double target2 = target * target;
    const int budget = gP.max_it - o.iterations;
    for (int it = 1; !converged && it <= budget; ++it) {
      // p = z + beta p, published; A: q = A p, (p, q)
      t0 = stamp();
      for_rows([&](int li, int row) {
        const double pn = d[li] * r[li] + beta * p[li];
        p[li] = pn;
        publish<double>(row, pn);
      });
      if (!exchange<double, 0>(part, red)) { o.aborted = 1; return; }
      part[0] = spmv<double>(gP.v64, [&](int li, int, double acc) {
        q[li] = acc;
        return p[li] * acc;
      });
      t1 = stamp();
      if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
      t2 = stamp();
      tm.a += t1 - t0;
      tm.aw += t2 - t1;
      const double pAp = red[0];
      const bool breakdown = (!continuation && gP.guard == 0) ? (fabs(pAp) < 1.0e-14)
                                                             : !(pAp > 0.0 && is_finite_d(pAp));
      if (breakdown) break;
      const double alpha = rz / pAp;
      // B: x += alpha p, r -= alpha q, (r, r), (r, z)
      t0 = t2;
      part[0] = part[1] = 0.0;
      for_rows([&](int li, int) {
        x[li] += alpha * p[li];
        const double rr = r[li] - alpha * q[li];
        r[li] = rr;
        part[0] += rr * rr;
        part[1] += rr * (d[li] * rr);
      });
      t1 = stamp();
      if (!S.template sums<2>(part, red)) { o.aborted = 1; return; }
      t2 = stamp();
      tm.b += t1 - t0;
      tm.bw += t2 - t1;
      ++o.iterations;
      double rz_new = red[1];
      est2 = red[0];
      const bool reached = est2 <= target2;
      if (S.late()) { o.status = FFG_TIMEOUT; break; }
      if (reached && !continuation) { converged = 1; break; }
      ++cycle_its;
      bool restart = false;
      if (continuation && (reached || (first_cycle > 0 && cycle_its >= 2 * first_cycle))) {
        t0 = stamp();
        if (first_cycle == 0) first_cycle = cycle_its;
        cycle_its = 0;
        restart = true;
        for_rows([&](int li, int row) { gP.x[row] = x[li]; });
        if (!barrier()) { o.aborted = 1; return; }
        part[0] = residual<false>(nullptr);
        if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
        true_res = sqrt(red[0]);
        est2 = red[0];
        if (true_res <= target) { converged = 1; tm.u += stamp() - t0; break; }
        stall = (true_res > 0.5 * last_true) ? stall + 1 : 0;
        last_true = true_res;
        if (stall >= 2 || !is_finite_d(true_res)) { tm.u += stamp() - t0; break; }
        ++o.updates;
        part[0] = 0.0;
        for_rows([&](int li, int row) {
          const double rr = gP.r64[row];
          r[li] = rr;
          part[0] += rr * (d[li] * rr);
        });
        if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
        tm.u += stamp() - t0;
        rz_new = red[0];
      }
      beta = (rz != 0.0 && !restart) ? rz_new / rz : 0.0;
      rz = rz_new;
    }
    o.converged = converged;
    o.final_res = sqrt(est2);
    // the solution, and its true FP64 residual
    t0 = stamp();
    if (rnorm > target) for_rows([&](int li, int row) { gP.x[row] = x[li]; });
    if (!barrier()) { o.aborted = 1; return; }
    part[0] = residual<false>(nullptr);
    if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
    tm.u += stamp() - t0;
    o.true_res = sqrt(red[0]);
  }

  // cg_mixed of kernels_pcg.cu.
  __device__ __forceinline__ void mixed(Outcome &o, Timing &tm) {
    setup<float>(gP.v32);
    float *r = vecs<float>(0), *p = vecs<float>(1), *q = vecs<float>(2), *d = vecs<float>(3),
          *xf = vecs<float>(4);
    double part[kVals] = {0, 0}, red[kVals];
    unsigned long long t0, t1, t2;
    t0 = stamp();
    if (!residual_norms(red)) { o.aborted = 1; return; }
    const double bnorm = sqrt(red[1]), rnorm = sqrt(red[0]);
    o.bnorm = bnorm;
    double scale = rnorm > 0.0 ? rnorm : 1.0;
    const double target = gP.relative ? gP.tol * bnorm : gP.tol;
    double true_res = rnorm, last_true = rnorm;
    int stall = 0, since = 0, window = kMinWindow;
    int converged = rnorm <= target ? 1 : 0;
    bool direct = false;
    double rz = 0.0;
    if (!converged) {
      const double inv = 1.0 / scale;
      part[0] = 0.0;
      for_rows([&](int li, int row) {
        const float rr = (float)(gP.r64[row] * inv), dd = gP.d32[row], zz = dd * rr;
        r[li] = rr;
        d[li] = dd;
        p[li] = 0.f;
        q[li] = 0.f;
        xf[li] = 0.f;
        publish<float>(row, zz);
        part[0] += (double)rr * (double)zz;
      });
      if (!exchange<float, 1>(part, red)) { o.aborted = 1; return; }
      rz = red[0];
    }
    tm.u += stamp() - t0;
    auto stop = [&]() {
      const double t = target / scale;
      return fmax(t * t, gP.delta * gP.delta);
    };
    double stop_rr = stop();
    double beta = 0.0;
    bool unfolded = false;  // xf holds a step not yet added to x
    auto fold = [&]() {
      for_rows([&](int li, int row) {
        gP.x[row] += (double)xf[li];
        xf[li] = 0.f;
      });
    };
    const int budget = gP.max_it - o.iterations;
    for (int it = 1; !converged && it <= budget; ++it) {
      // A: q = A p, p = z + beta p, (p, q)
      t0 = stamp();
      const float bt = (float)beta;
      if (!direct) {
        part[0] = spmv<float>(gP.v32, [&](int li, int, float acc) {
          const float pn = d[li] * r[li] + bt * p[li];
          const float qn = acc + bt * q[li];
          p[li] = pn;
          q[li] = qn;
          return (double)pn * (double)qn;
        });
      } else {
        for_rows([&](int li, int row) {
          const float pn = d[li] * r[li] + bt * p[li];
          p[li] = pn;
          publish<float>(row, pn);
        });
        if (!exchange<float, 0>(part, red)) { o.aborted = 1; return; }
        part[0] = spmv<float>(gP.v32, [&](int li, int, float acc) {
          q[li] = acc;
          return (double)p[li] * (double)acc;
        });
      }
      t1 = stamp();
      if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
      t2 = stamp();
      tm.a += t1 - t0;
      tm.aw += t2 - t1;
      const double pAp = red[0];
      if (!(pAp > 0.0 && is_finite_d(pAp))) {
        o.stagnated = 1;
        o.restart = 1;
        break;
      }
      const double alpha = rz / pAp;
      const float al = (float)alpha;
      const float xs = (float)(alpha * scale);
      // B: dx += alpha p, r -= alpha q, z = D^-1 r
      t0 = t2;
      part[0] = part[1] = 0.0;
      for_rows([&](int li, int row) {
        xf[li] += xs * p[li];
        const float rr = r[li] - al * q[li];
        r[li] = rr;
        const float zz = d[li] * rr;
        if (!direct) publish<float>(row, zz);
        part[0] += (double)rr * (double)rr;
        part[1] += (double)rr * (double)zz;
      });
      t1 = stamp();
      if (!(direct ? S.template sums<2>(part, red) : exchange<float, 2>(part, red))) {
        o.aborted = 1;
        return;
      }
      t2 = stamp();
      tm.b += t1 - t0;
      tm.bw += t2 - t1;
      ++o.iterations;
      unfolded = true;
      const double rr = red[0], rz_new = red[1];
      if (S.late()) {
        o.status = FFG_TIMEOUT;
        true_res = sqrt(rr) * scale;
        break;
      }
      // the estimate sqrt(rr) * scale against the target, delta and growth, squared
      const bool grew = !(rr < 100.0);
      const bool slow = o.iterations - since > window;
      if (!(rr <= stop_rr || grew || slow)) {
        beta = rz_new / rz;
        rz = rz_new;
        continue;
      }
      if (o.updates >= gP.max_updates) break;
      ++o.updates;
      t0 = stamp();
      fold();
      // x becomes visible, and the copies of z have landed everywhere
      if (IDX == kAbs16 && !barrier()) { o.aborted = 1; return; }
      if (!direct) {
        for_rows([&](int li, int row) { publish<float>(row, p[li]); });
        if (IDX == kAbs16 && !exchange<float, 0>(part, red)) { o.aborted = 1; return; }
      }
      if (IDX != kAbs16 && !barrier()) { o.aborted = 1; return; }
      unfolded = false;
      part[0] = direct ? residual<false>(nullptr) : residual<true>(q);
      if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
      true_res = sqrt(red[0]);
      if (true_res <= target) { converged = 1; tm.u += stamp() - t0; break; }
      if (!(true_res > 0.0) || !is_finite_d(true_res)) break;
      stall = (true_res > 0.5 * last_true) ? stall + 1 : 0;
      last_true = true_res;
      if (stall >= 2) { o.stagnated = 1; tm.u += stamp() - t0; break; }
      if (!direct && (slow || (stall > 0 && !grew))) direct = true;
      const double ratio = scale / true_res;
      const double inv = 1.0 / true_res;
      part[0] = 0.0;
      for_rows([&](int li, int row) {
        const float rr2 = (float)(gP.r64[row] * inv);
        const float zz = d[li] * rr2;
        r[li] = rr2;
        if (!direct) publish<float>(row, zz);
        part[0] += (double)rr2 * (double)zz;
      });
      if (!(direct ? S.template sums<1>(part, red) : exchange<float, 1>(part, red))) {
        o.aborted = 1;
        return;
      }
      tm.u += stamp() - t0;
      beta = grew ? 0.0 : red[0] / (rz * ratio);
      rz = red[0];
      scale = true_res;
      stop_rr = stop();
      window = max(kMinWindow, 4 * (o.iterations - since));
      since = o.iterations;
    }
    if (unfolded) {
      fold();
      if (!barrier()) { o.aborted = 1; return; }
    }
    o.converged = converged;
    o.final_res = true_res;
    if (converged) {
      o.true_res = true_res;
      return;
    }
    if (o.stagnated) return;  // the FP64 continuation measures its own residual
    t0 = stamp();
    part[0] = residual<false>(nullptr);
    if (!S.template sums<1>(part, red)) { o.aborted = 1; return; }
    tm.u += stamp() - t0;
    o.true_res = sqrt(red[0]);
    o.final_res = o.true_res;
  }

  __device__ __forceinline__ void init(const Share &h, const Sync &sync) {
    S = sync;
    const unsigned tab_bytes = (unsigned)((h.tab_slices * sizeof(SliceEnt) + 127) & ~(size_t)127);
    tab = reinterpret_cast<SliceEnt *>(res_pool);
    pool = res_pool + tab_bytes;
    pool_bytes = h.pool_bytes - tab_bytes;
    s0 = h.s0;
    nsl = h.nsl;
    R = nsl * kSliceRows;
    tid = threadIdx.x;
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    // Columns of a part: small enough that the slices spread over the warps,
    // whole slices where there are many of them a warp, and more where the
    // items and their scratch would not fit (P4, 132,651 rows: whole slices
    // there cost one CTA 37 us where the others took 12).  Items in slice
    // order, at the pool's end (its start holds the published vector's replica).
    for (int i = tid; i < nsl; i += NT) {
      const int s = s0 + i;
      const int64_t g = gP.soff[s];
      tab[i] = SliceEnt{g, -1, (int)((gP.soff[s + 1] - g) / kSliceRows), 0, 1, 0};
    }
    for (int chunk = nsl >= 2 * (NT / 32) ? 32 : 16;; chunk *= 2) {
      const bool last = chunk > kMaxColumnLength;
      for (int i = tid; i < nsl; i += NT) {
        const int len = tab[i].len;
        const int parts = last || len <= chunk + chunk / 4 ? 1 : (len + chunk - 1) / chunk;
        tab[i].parts = parts;
        tab[i].cols = parts == 1 ? len : ((len + parts - 1) / parts + kBatch - 1) / kBatch * kBatch;
      }
      __syncthreads();
      if (warp == 0) {
        int sum = 0, rows = 0;
        for (int i0 = 0; i0 < nsl; i0 += 32) {
          const int i = i0 + lane, e = i < nsl ? tab[i].parts : 0, m = e > 1 ? e : 0;
          int x = e, y = m;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, x, o), b = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) {
              x += a;
              y += b;
            }
          }
          if (i < nsl) {
            tab[i].off = sum + x - e;  // first item, until setup
            tab[i].part0 = rows + y - m;
          }
          sum += __shfl_sync(0xffffffffu, x, 31);
          rows += __shfl_sync(0xffffffffu, y, 31);
        }
        if (lane == 0) {
          gSh.items = sum;
          gSh.rows = rows;
        }
      }
      __syncthreads();
      items = gSh.items;
      scratch_rows = gSh.rows;
      const size_t extra = (size_t)(items - nsl) * sizeof(unsigned) +
                           (size_t)scratch_rows * 32 * sizeof(double2);
      if (last || extra <= h.part_bytes) break;
      __syncthreads();
    }
    const unsigned bytes = (unsigned)((items * sizeof(unsigned) + 127) & ~(size_t)127);
    pool_bytes = (pool_bytes - bytes) & ~127u;
    item = reinterpret_cast<unsigned *>(pool + pool_bytes);
    for (int i = tid; i < nsl; i += NT)
      for (int k = 0; k < tab[i].parts; ++k) item[tab[i].off + k] = (unsigned)i | (unsigned)k << 16;
    __syncthreads();
  }
};

template <class Sync, int IDX, int NT>
__device__ __noinline__ Sync run_mixed(Share h, Sync sync, Outcome &out, Timing &tmo) {
  Solve<Sync, IDX, NT> X;
  X.init(h, sync);
  Outcome o;
  Timing tm;
  X.mixed(o, tm);
  out = o;
  tmo = tm;
  return X.S;
}

template <class Sync, int IDX, int NT>
__device__ __noinline__ Sync run_fp64(Share h, Sync sync, bool continuation, Outcome &out, Timing &tmo) {
  Solve<Sync, IDX, NT> X;
  X.init(h, sync);
  Outcome o = out;
  Timing tm = tmo;
  if (continuation && o.restart) {
    X.for_rows([&](int, int row) { gP.x[row] = 0.0; });
  }
  if (!X.barrier()) o.aborted = 1;
  else X.fp64(continuation, o, tm);
  out = o;
  tmo = tm;
  return X.S;
}

// The whole solve of gP by the CTAs of `sync`.  gP.staged: bit 0, the mixed
// loop's published vector fits the shared-memory pool of every CTA (bit 1: the
// FP64 loop's).
template <class Sync, bool kShared, int NT>
__device__ __forceinline__ void run_solve(const Share &h, Sync sync) {
  const unsigned long long t_start = globaltimer(), c_start = clock_now();
  if (threadIdx.x == 0) {
    gSh.deadline = t_start + gP.limit_ns;
    gSh.past_limit = 0;
  }
  Outcome o;
  Timing tm;
  int continued = 0;
  bool fp64 = gP.precision == FFG_PRECISION_FP64, continuation = false;
  if (!fp64) {
    bool done = false;
    if constexpr (kShared) {
      if (gP.staged & 1) {
        sync = run_mixed<Sync, kAbs16, NT>(h, sync, o, tm);
        done = true;
      }
    }
    if (done) {
    } else if (gP.dcol) sync = run_mixed<Sync, kRel16, NT>(h, sync, o, tm);
    else sync = run_mixed<Sync, kAbs32, NT>(h, sync, o, tm);
    if (!o.aborted && o.stagnated && !o.converged && o.status == FFG_OK) {
      continued = o.restart ? 2 : 1;
      fp64 = continuation = true;
    }
  }
  if (fp64 && !o.aborted) {
    bool done = false;
    if constexpr (kShared) {
      if (gP.staged & 2) {
        run_fp64<Sync, kAbs16, NT>(h, sync, continuation, o, tm);
        done = true;
      }
    }
    if (done) {
    } else if (gP.dcol) run_fp64<Sync, kRel16, NT>(h, sync, continuation, o, tm);
    else run_fp64<Sync, kAbs32, NT>(h, sync, continuation, o, tm);
  }
  if (o.aborted) {
    // a sync gave up: the host reads the status, not an older result
    if (threadIdx.x == 0) atomicCAS(gP.control, 0, FFG_TIMEOUT);
    if (sync.rank == 0 && threadIdx.x == 0) {
      gP.result[0] = 0.0;
      gP.result[5] = FFG_TIMEOUT;
    }
    return;
  }
  if (sync.rank == 0 && threadIdx.x == 0) {
    const double c = (double)(clock_now() - c_start);
    const double sec = c > 0.0 ? 1e-9 * (double)(globaltimer() - t_start) / c : 0.0;
    gP.result[0] = o.converged;
    gP.result[1] = o.iterations;
    gP.result[2] = o.updates;
    gP.result[3] = o.final_res;
    gP.result[4] = o.bnorm > 0.0 ? o.true_res / o.bnorm : o.true_res;
    gP.result[5] = o.status;
    gP.result[6] = o.bnorm;
    gP.result[7] = continued;
    gP.result[8] = sec * (double)tm.a;
    gP.result[9] = sec * (double)tm.aw;
    gP.result[10] = sec * (double)tm.b;
    gP.result[11] = sec * (double)tm.bw;
    gP.result[12] = sec * (double)tm.u;
  }
}

constexpr int kMaxClusterBatch = 48;
struct ClusterBatch {
  PcgParams sys[kMaxClusterBatch];
};

// Cluster c solves sys[c]; its CTAs take the slice ranges gP.cta_slice.
template <int NT>
__global__ void __launch_bounds__(NT, 1) pcg_cluster_kernel(const __grid_constant__ ClusterBatch B) {
  // a launch of this kernel may follow another one of the same batch at once
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  unsigned rank, size;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %cluster_nctarank;" : "=r"(size));
  if (threadIdx.x == 0) {
    gP = B.sys[blockIdx.x / size];
    gSh.ok = 1;
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&gSh.mbar[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&gSh.mbar_all[i])), "r"(size));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (rank == 0) gP.control[0] = 0;  // as every launch begins, before any CTA's first wait
  }
  __syncthreads();
  const int C = (int)size, r = (int)rank, s0 = gP.cta_slice[r];
  const Share h{s0, gP.cta_slice[r + 1] - s0, gP.share_slices, kPoolMax, (unsigned)gP.part_bytes};
  ClusterSync<NT> S{r, C, 0u, 0u};
  S.rendezvous();  // every CTA's mbarriers are ready
  run_solve<ClusterSync<NT>, true, NT>(h, S);
  S.rendezvous();  // no CTA leaves while others may still store into it
  // A wait that gave up may have left messages under way, all of them sent
  // before the rendezvous: time for them to land.
  if (threadIdx.x == 0 && ld_volatile_int(gP.control) != 0)
    for (const unsigned long long t0 = globaltimer(); globaltimer() - t0 < kLandNs;) __nanosleep(1000);
  // what comes after this launch comes after the launch it overlapped with too
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The whole cooperative grid solves one system; CTAs take the contiguous slice
// ranges of the operator's partition.
__global__ void __launch_bounds__(kGridThreads, 1)
    pcg_resident_kernel(const __grid_constant__ PcgParams P, unsigned pool_bytes) {
  if (threadIdx.x == 0) {
    gP = P;
    gSh.ok = 1;
  }
  __syncthreads();
  const int c = (int)blockIdx.x, s0 = gP.cta_slice[c];
  const int nsl = gP.cta_slice[c + 1] - s0;
  const Share h{s0, nsl, nsl, pool_bytes, (unsigned)gP.part_bytes};
  using Sync = GridSync<kGridThreads, false>;
  run_solve<Sync, false, kGridThreads>(h, Sync{c, gP.ncta, 0u});
}

// Slice where CTA r of a group of G starts: equal cost, a slice costing its
// entries and kGroupSliceCost for its rows.
constexpr int kGroupSliceCost = 256;
__host__ __device__ inline int group_cut(const int64_t *soff, int64_t n_slices, int r, int G) {
  const int64_t target =
      (soff[n_slices] + (int64_t)kGroupSliceCost * n_slices) * (int64_t)r / G;
  int64_t lo = 0, hi = n_slices;  // first slice whose cost before it reaches the target
  while (lo < hi) {
    const int64_t m = (lo + hi) / 2;
    if (soff[m] + (int64_t)kGroupSliceCost * m < target) lo = m + 1;
    else hi = m;
  }
  return r >= G ? (int)n_slices : (int)lo;
}

// Several systems in one cooperative launch, system i on CTAs first[i] ..
// first[i + 1] - 1.  A group's sync waits only on its own CTAs, which the launch
// makes resident together.
struct GroupBatch {
  PcgParams sys[kMaxResidentGroups];
  int first[kMaxResidentGroups + 1];
  int count;
};
__global__ void __launch_bounds__(kGridThreads, 1)
    pcg_resident_group_kernel(const __grid_constant__ GroupBatch B) {
  int i = 0;
  while (i + 1 < B.count && B.first[i + 1] <= (int)blockIdx.x) ++i;
  if (threadIdx.x == 0) {
    gP = B.sys[i];
    gSh.ok = 1;
  }
  __syncthreads();
  const int c = (int)blockIdx.x - B.first[i];
  const int s0 = group_cut(gP.soff, gP.n_slices, c, gP.ncta);
  const int nsl = group_cut(gP.soff, gP.n_slices, c + 1, gP.ncta) - s0;
  const Share h{s0, nsl, nsl, kPoolMax, (unsigned)gP.part_bytes};
  using Sync = GridSync<kGridThreads, true>;
  run_solve<Sync, false, kGridThreads>(h, Sync{c, gP.ncta, 0u});
}

// Shared memory beside the operator: the slice and item tables, five vectors
// of the CTA's rows and the published vector when it is replicated.
size_t fixed_bytes(int64_t slices_per_cta, int64_t n_slices, int elem, bool replica) {
  const size_t rows = (size_t)slices_per_cta * kSliceRows;
  return ((size_t)slices_per_cta * (sizeof(SliceEnt) + sizeof(unsigned)) + 255) / 128 * 128 +
         (5 * rows * elem + 127) / 128 * 128 +
         (replica ? (size_t)n_slices * (kSliceRows * elem + 1) + 255 : 0) / 128 * 128 +
         1024;
}

// Largest cluster of pcg_cluster_kernel this device takes (16, 8 or 0), with
// the kernels opted into kPoolMax bytes of dynamic shared memory (once per device).
int resident_ready() {
  static std::mutex mu;
  static int state[64] = {0};  // 0 unknown, -1 refused, else the cluster size
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return 0;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (state[dev] == 0) {
    state[dev] = -1;
    bool ok = true;
    for (const void *f : {(const void *)pcg_resident_kernel, (const void *)pcg_resident_group_kernel})
      ok = ok && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kPoolMax) ==
                     cudaSuccess;
    int top = kMaxCluster;
    auto cluster_kernel = [&](auto kern, int threads) {
      ok = ok &&
           cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kPoolMax) == cudaSuccess &&
           cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                1) == cudaSuccess;
      for (; ok && top >= 8; top /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(top);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = kPoolMax;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = top;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0)
          break;
      }
    };
    cluster_kernel(pcg_cluster_kernel<256>, 256);
    cluster_kernel(pcg_cluster_kernel<512>, 512);
    if (ok && top >= 8) state[dev] = top;
    cudaGetLastError();
  }
  return std::max(state[dev], 0);
}

int cluster_index(int c) { return c == 16 ? 1 : 0; }

// Bytes of a CTA's largest share beside the operator, over the loops a solve
// of this precision may run (the FP64 continuation of a mixed solve may leave
// its published vector in global memory).
size_t loops_bytes(int64_t slices, int64_t n_slices, bool fp64, bool replica) {
  return std::max(fixed_bytes(slices, n_slices, fp64 ? 8 : 4, replica),
                  fixed_bytes(slices, n_slices, 8, replica && fp64));
}
}  // namespace

size_t pcg_message_bytes(int ctas) { return 2 * (size_t)ctas * 32; }

// Lines between the kernels, measured on a B200 (solve time of P1, P2 and
// order-1 Nedelec systems, clusters of 16 against the whole grid):
//  mixed, P2:       12,167 rows, 307 k entries 1.33 / 1.87 ms;
//  mixed, Nedelec:  21,645 rows, 332 k entries 4.79 / 5.69 ms;
//  mixed, P1:       28,561 rows, 199 k entries 4.57 / 7.70 ms; 39,601 rows,
//                   276 k entries (60 KB of a CTA's operator from L2) 8.10 / 10.6 ms;
//  FP64, P2:        6,859 rows, 168 k entries 1.00 / 1.48 ms; 12,167 rows,
//                   307 k entries 1.84 / 1.77 ms;
//  FP64, P1:        19,321 rows, 134 k entries 4.14 / 6.42 ms.
// In a cluster an entry costs shared-memory bandwidth on 16 SMs, on the grid
// a sync costs three to four times the cluster's.  In a batch the other choice
// is one CTA, so only the fit decides; systems below 10,000 rows + entries / 11
// take 8 CTAs there (P1, 1,521 rows: 0.55 ms with 8 and with 16; 19,321 rows:
// 4.4 / 3.2 ms), which leaves SMs to the others.
int pcg_cluster_size(const DeviceSell &A, int precision, bool batched) {
  if (precision == FFG_PRECISION_MIXED16 || A.n < 1 || !A.cluster_slice) return 0;
  const int top = resident_ready();
  if (!top) return 0;
  const bool fp64 = precision == FFG_PRECISION_FP64;
  const int c = batched && 11 * A.n + A.padded <= 110000 ? 8 : top;
  const int64_t per = A.cluster_share[cluster_index(c)];
  const size_t fixed = loops_bytes(per, A.n_slices, fp64, true);
  if (fixed > (size_t)kPoolMax) return 0;
  if (batched) return c;
  return A.padded <= (fp64 ? 280000 : 450000) ? c : 0;
}

// The grid kernel where the operator fits the chip, and beyond that while it
// stays in L2 between iterations (resident part + L2, solve time against the
// staged kernel): P2, 250,047 rows, FP64 (69 MB) 14.3 / 16.5 ms, 357,911 rows
// mixed (59 MB) 14.4 / 16.0, FP64 (98 MB) 35 / 23; 493,039 rows mixed (82 MB)
// 21.1 / 19.9.  The staged kernel gives a slice to one warp of 32, so with
// fewer slices a CTA than that the line lies higher: P4, 132,651 rows, mixed
// (55 MB) 20.0 / 37.5 ms, FP64 (91 MB) 39 / 64.
constexpr size_t kGridL2Bytes = 75000000, kGridL2BytesFew = 95000000;

size_t pcg_grid_resident(const DeviceSell &A, int precision) {
  if (precision == FFG_PRECISION_MIXED16 || A.n < 1 || A.grid > 32 * kPoll) return 0;
  if (!resident_ready()) return 0;
  const bool fp64 = precision == FFG_PRECISION_FP64;
  const size_t fixed = loops_bytes(A.share_slices, A.n_slices, fp64, false);
  if (fixed > (size_t)kPoolMax) return 0;
  // the operator as this precision's loop keeps it, and, where rows are long
  // enough to be split, about a quarter more for their parts
  size_t need = (size_t)A.share_entries * ((fp64 ? 8 : 4) + (A.dcol ? 2 : 4));
  if (A.padded > 16 * A.n) need += need / 4;
  need = std::max(fixed, need + fixed_bytes(A.share_slices, A.n_slices, fp64 ? 8 : 4, false));
  const size_t bytes = (size_t)A.padded * ((fp64 ? 8 : 4) + (A.dcol ? 2 : 4));
  if (need > (size_t)kPoolMax &&
      bytes > (A.n_slices > (int64_t)32 * A.grid ? kGridL2Bytes : kGridL2BytesFew))
    return 0;
  return std::min<size_t>((need + 1023) & ~(size_t)1023, kPoolMax);
}

int pcg_group_shape(const DeviceSell &A, int precision, int grid, int *max_slices) {
  if (precision == FFG_PRECISION_MIXED16 || A.n < 1 || grid > 32 * kPoll ||
      (int64_t)A.host_soff.size() != A.n_slices + 1 || !resident_ready())
    return 0;
  const bool fp64 = precision == FFG_PRECISION_FP64;
  const size_t entry = (fp64 ? 8 : 4) + (A.dcol ? 2 : 4);
  const int64_t *soff = A.host_soff.data();
  // a k-th of the grid each, so that groups fill it: the largest k (of at most
  // kMaxResidentGroups) whose CTAs hold the operator but for a twelfth
  for (int k = std::min(kMaxResidentGroups, grid / 2); k >= 1; --k) {
    const int G = grid / k;
    int64_t entries = 0;
    int slices = 0;
    for (int r = 0, s0 = 0; r < G; ++r) {
      const int s1 = group_cut(soff, A.n_slices, r + 1, G);
      slices = std::max(slices, s1 - s0);
      entries = std::max(entries, soff[s1] - soff[s0]);
      s0 = s1;
    }
    const size_t fixed = loops_bytes(slices, A.n_slices, fp64, false);
    if (fixed <= (size_t)kPoolMax &&
        fixed + (size_t)entries * entry <= (size_t)kPoolMax + kPoolMax / 12) {
      *max_slices = slices;
      return G;
    }
  }
  return 0;
}

cudaError_t pcg_launch_resident_groups(int count, const PcgParams *sys, cudaStream_t s) {
  static_assert(sizeof(GroupBatch) <= 32000, "kernel parameter block too large");
  GroupBatch B;
  B.count = count;
  B.first[0] = 0;
  for (int i = 0; i < count; ++i) {
    PcgParams &P = B.sys[i];
    P = sys[i];
    const size_t fixed =
        loops_bytes(P.share_slices, P.n_slices, P.precision == FFG_PRECISION_FP64, false);
    P.part_bytes = (int)std::min<size_t>(kPoolMax / 8, kPoolMax - fixed);
    B.first[i + 1] = B.first[i] + P.ncta;
  }
  void *args[] = {&B};
  return cudaLaunchCooperativeKernel((const void *)pcg_resident_group_kernel,
                                     dim3(B.first[count]), dim3(kGridThreads), args, kPoolMax, s);
}

cudaError_t pcg_launch_cluster(int count, const PcgParams *sys, int cluster, bool batched,
                               bool overlap, cudaStream_t s) {
  static_assert(sizeof(ClusterBatch) <= 32000, "kernel parameter block too large");
  ClusterBatch B;
  for (int c0 = 0; c0 < count; c0 += kMaxClusterBatch) {
    const int m = std::min(kMaxClusterBatch, count - c0);
    int per = 0;
    for (int i = 0; i < m; ++i) {
      PcgParams &P = B.sys[i];
      P = sys[c0 + i];
      P.ncta = cluster;
      P.cta_slice = P.cluster_slice + (cluster_index(cluster) ? 9 : 0);
      P.share_slices = P.cluster_share[cluster_index(cluster)];
      per = std::max(per, P.share_slices);
      P.staged = 0;
      for (int k = 0; k < 2; ++k)
        if (fixed_bytes(P.share_slices, P.n_slices, 4 << k, true) <= (size_t)kPoolMax)
          P.staged |= 1 << k;
      const size_t fixed = std::max(
          loops_bytes(P.share_slices, P.n_slices, P.precision == FFG_PRECISION_FP64, true),
          (P.staged & 2) ? fixed_bytes(P.share_slices, P.n_slices, 8, true) : 0);
      P.part_bytes = (int)std::min<size_t>(kPoolMax / 8, kPoolMax - fixed);
    }
    // 256 threads shorten the sums while a thread has few rows; a batch takes
    // one block size, so that a system's result does not depend on the others
    const int threads = !batched && per <= 16 ? 256 : 512;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(m * cluster);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = kPoolMax;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap || c0 > 0 ? 2 : 1;
    const cudaError_t e = threads == 256 ? cudaLaunchKernelEx(&cfg, pcg_cluster_kernel<256>, B)
                                         : cudaLaunchKernelEx(&cfg, pcg_cluster_kernel<512>, B);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t pcg_launch_resident(const PcgParams &P, size_t pool_bytes, cudaStream_t s) {
  PcgParams Q = P;
  unsigned pool = (unsigned)pool_bytes;
  const size_t fixed =
      loops_bytes(P.share_slices, P.n_slices, P.precision == FFG_PRECISION_FP64, false);
  Q.part_bytes = (int)std::min<size_t>(pool_bytes / 8, pool_bytes - fixed);
  void *args[] = {&Q, &pool};
  return cudaLaunchCooperativeKernel((const void *)pcg_resident_kernel, dim3(P.ncta),
                                     dim3(kGridThreads), args, pool, s);
}

}  // namespace ffg
