// The messages of one phase of a cluster's sums (kernels_pcg_resident.cu).
//
// Phase k uses slot set and mbarrier k % 2 of every CTA.  A CTA may send into
// them again in phase k + 2, which it starts once phase k + 1 has completed at
// it; if every CTA sends to every CTA in every phase, all have then started
// phase k + 1, so they have read their slots of phase k and finished its wait.  A phase
// without sums therefore sends a message that nobody reads: one that waited
// for the copied slices alone would let a CTA that reads none of another's run
// two phases ahead of it.
#pragma once

#ifdef __CUDACC__
#define FFG_HOST_DEVICE __host__ __device__
#else
#define FFG_HOST_DEVICE
#endif

namespace ffg {

// 8-byte messages that each CTA sends to each CTA in a phase of nv sums.
FFG_HOST_DEVICE constexpr int phase_messages(int nv) { return nv > 0 ? nv : 1; }

// Bytes that a CTA's mbarrier expects in it: the messages of n CTAs and the
// slices copied to it.
FFG_HOST_DEVICE constexpr unsigned phase_bytes(int nv, int n, unsigned copied) {
  return 8u * (unsigned)(phase_messages(nv) * n) + copied;
}

}  // namespace ffg
