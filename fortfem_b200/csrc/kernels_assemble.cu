// Assembly kernels (sm_100a): per-cell geometry (K1), Nedelec element
// matrices with orientation transform (K2), and the atomic-free,
// column-owner scatter into the constrained CSC (K3).
//
// K3 gives every CSC column (a free global DoF j) to one thread, or to a group
// of lanes (the slice gather below), which works in the same order.  The thread
// walks the cells incident to j in ascending cell order, computes column l(j)
// of each element matrix and adds it into the column's slots through the
// precomputed slot map.  Every CSC value is therefore the sum of its element
// contributions in the reference's triplet order (cell-major, as
// assemble_*_csc emits them before csc_from_triplet), without atomics, and is
// bit-reproducible run to run.  The same pass accumulates the load, the
// Dirichlet lifting -A_fc g of sparse_direct_solve_constrained_real
// (src/solvers/fortfem_sparse_direct.f90:329-338, by symmetry of the element
// matrices) and the Jacobi diagonal of build_sparse_preconditioner
// (src/solvers/advanced_solvers.f90:1139-1154).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "ffg_internal.h"
#include "tet_geometry.h"

namespace ffg {

namespace {

// symmetric pair order shared with basis.cpp: (0,0),(1,1),(2,2),(0,1),(0,2),(1,2)
__constant__ int kPa[6] = {0, 1, 2, 0, 0, 1};
__constant__ int kPb[6] = {0, 1, 2, 1, 2, 2};

// ------------------------------------------------------------ K1 geometry
// Lagrange: geo = [k det G_ab (6), m det, det f_q (n_q)], G = J^-1 J^-T.
__device__ __forceinline__ void lagrange_geometry_cell(int c, const int *__restrict__ cells,
                                                      const double *__restrict__ verts, double ca,
                                                      double cb, const double *__restrict__ cell_a,
                                                      const double *__restrict__ cell_b,
                                                      const double *__restrict__ samples, int nq,
                                                      double *__restrict__ geo, int stride,
                                                      int *err) {
  double J[9], Ji[9], v0[3];
  tet_jacobian(cells, verts, c, J, v0);
  const double det = det3(J);
  double *g = geo + (size_t)stride * c;
  if (!valid_jacobian(J, det)) {
    atomicCAS(err, 0, FFG_INVALID_INPUT);
    for (int i = 0; i < stride; ++i) g[i] = 0.0;
    return;
  }
  inv3(J, det, Ji);
  const double kappa = ca * (cell_a ? cell_a[c] : 1.0);
  const double mass = cb * (cell_b ? cell_b[c] : 1.0);
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    const int a = kPa[s], b = kPb[s];
    // (J^-1 J^-T)_ab = sum_k Ji(a,k) Ji(b,k), Ji column-major Ji[a + 3k]
    const double G = Ji[a] * Ji[b] + Ji[a + 3] * Ji[b + 3] + Ji[a + 6] * Ji[b + 6];
    g[s] = kappa * det * G;
  }
  g[6] = mass * det;
  for (int q = 0; q < nq; ++q) g[7 + q] = samples ? det * samples[(size_t)nq * c + q] : 0.0;
}

__global__ void lagrange_geometry_kernel(int n_cells, const int *__restrict__ cells,
                                         const double *__restrict__ verts, double ca, double cb,
                                         const double *__restrict__ cell_a,
                                         const double *__restrict__ cell_b,
                                         const double *__restrict__ samples, int nq,
                                         double *__restrict__ geo, int stride, int *err) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n_cells)
    lagrange_geometry_cell(c, cells, verts, ca, cb, cell_a, cell_b, samples, nq, geo, stride, err);
}

// P1 triangles: closed-form local matrix of assemble_scalar_p1_matrix
// (src/fortfem_forms_simple.f90:1702-1717) and the load area/3 of
// assemble_scalar_p1_load (:1749-1758) with a per-cell source value.
__device__ __forceinline__ void p1_geometry_cell(int c, const int *__restrict__ tris,
                                                 const double *__restrict__ verts, double stiff,
                                                 double mass, const double *__restrict__ cell_a,
                                                 const double *__restrict__ cell_b,
                                                 const double *__restrict__ samples,
                                                 double *__restrict__ geo, int *err) {
  double x[3], y[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int v = tris[3 * (size_t)c + i];
    x[i] = verts[2 * (size_t)v];
    y[i] = verts[2 * (size_t)v + 1];
  }
  const double det = (x[1] - x[0]) * (y[2] - y[0]) - (x[2] - x[0]) * (y[1] - y[0]);
  double *g = geo + 10 * (size_t)c;
  if (fabs(det) <= 64.0 * kEps) {
    atomicCAS(err, 0, FFG_INVALID_INPUT);
    for (int i = 0; i < 10; ++i) g[i] = 0.0;
    return;
  }
  const double area = 0.5 * fabs(det);
  const double gx[3] = {(y[1] - y[2]) / det, (y[2] - y[0]) / det, (y[0] - y[1]) / det};
  const double gy[3] = {(x[2] - x[1]) / det, (x[0] - x[2]) / det, (x[1] - x[0]) / det};
  const double ks = stiff * (cell_a ? cell_a[c] : 1.0);
  const double km = mass * (cell_b ? cell_b[c] : 1.0);
#pragma unroll
  for (int b = 0; b < 3; ++b)
#pragma unroll
    for (int a = 0; a < 3; ++a)
      g[a + 3 * b] = ks * area * (gx[a] * gx[b] + gy[a] * gy[b]) +
                     km * area * (a == b ? 2.0 : 1.0) / 12.0;
  g[9] = samples ? samples[c] * area / 3.0 : 0.0;
}

__global__ void p1_geometry_kernel(int n_cells, const int *__restrict__ tris,
                                   const double *__restrict__ verts, double stiff, double mass,
                                   const double *__restrict__ cell_a,
                                   const double *__restrict__ cell_b,
                                   const double *__restrict__ samples, double *__restrict__ geo,
                                   int *err) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n_cells) p1_geometry_cell(c, tris, verts, stiff, mass, cell_a, cell_b, samples, geo, err);
}

// Arbitrary-order triangles: geo = [k |det| G_00, k |det| G_11, k |det| G_01,
// m |det|, |det| f_q (n_q)], G = J^-1 J^-T of the affine map (columns v1 - v0,
// v2 - v0); |det| as the P1 forms take the unsigned area.
__global__ void triangle_lagrange_geometry_kernel(int n_cells, const int *__restrict__ tris,
                                                  const double *__restrict__ verts, double ca,
                                                  double cb, const double *__restrict__ cell_a,
                                                  const double *__restrict__ cell_b,
                                                  const double *__restrict__ samples, int nq,
                                                  double *__restrict__ geo, int stride, int *err) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cells) return;
  double x[3], y[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int v = tris[3 * (size_t)c + i];
    x[i] = verts[2 * (size_t)v];
    y[i] = verts[2 * (size_t)v + 1];
  }
  const double j00 = x[1] - x[0], j10 = y[1] - y[0], j01 = x[2] - x[0], j11 = y[2] - y[0];
  const double det = j00 * j11 - j01 * j10;
  const double m = fmax(fmax(fabs(j00), fabs(j10)), fmax(fabs(j01), fabs(j11)));
  const double sc = fmax(1.0, m);
  double *g = geo + (size_t)stride * c;
  if (!(fabs(det) > 64.0 * kEps * sc * sc)) {
    atomicCAS(err, 0, FFG_INVALID_INPUT);
    for (int i = 0; i < stride; ++i) g[i] = 0.0;
    return;
  }
  // J^-1 rows: (j11, -j01) / det and (-j10, j00) / det
  const double i00 = j11 / det, i01 = -j01 / det, i10 = -j10 / det, i11 = j00 / det;
  const double area = fabs(det);
  const double kappa = ca * (cell_a ? cell_a[c] : 1.0);
  const double mass = cb * (cell_b ? cell_b[c] : 1.0);
  g[0] = kappa * area * (i00 * i00 + i01 * i01);
  g[1] = kappa * area * (i10 * i10 + i11 * i11);
  g[2] = kappa * area * (i00 * i10 + i01 * i11);
  g[3] = mass * area;
  for (int q = 0; q < nq; ++q) g[4 + q] = samples ? area * samples[(size_t)nq * c + q] : 0.0;
}

// ----------------------------------------------------- K3 column-owner scatter
// SELL = false: values into the CSC value array (rhs in free-DoF order).
// SELL = true: values into the solver's slices (row iperm[j] of the SELL
// operator, which by symmetry is column j), with the FP32 copy, the Jacobi
// diagonal and the rhs in the SELL numbering.
template <int FAMILY, bool SELL>
__device__ __forceinline__ void column_body(int64_t j, const int64_t *__restrict__ col_ptr,
                              const int *__restrict__ row_idx, const int64_t *__restrict__ inc_ptr,
                              const int *__restrict__ inc_cell,
                              const uint8_t *__restrict__ inc_local,
                              const uint16_t *__restrict__ slot, const int *__restrict__ gd,
                              int nb, const double *__restrict__ geo, int stride,
                              const double *__restrict__ ref, const double *__restrict__ load_basis,
                              int nq, const double *__restrict__ elem,
                              const double *__restrict__ cell_rhs, const double *__restrict__ g,
                              const int *__restrict__ iperm, const int64_t *__restrict__ soff,
                              double *__restrict__ val64, float *__restrict__ val32,
                              double *__restrict__ dinv64, float *__restrict__ dinv32,
                              double *__restrict__ rhs, const float *__restrict__ elem32,
                              int ld32, int64_t cs32) {
  const int64_t start = col_ptr[j], end = col_ptr[j + 1];
  int64_t base, stride_out, out_row;
  if (SELL) {
    out_row = iperm[j];
    base = soff[out_row / kSliceRows] + out_row % kSliceRows;
    stride_out = kSliceRows;
  } else {
    out_row = j;
    base = start;
    stride_out = 1;
  }
  const int len = (int)(end - start);
  for (int k = 0; k < len; ++k) val64[base + stride_out * k] = 0.0;
  double b = 0.0, lift = 0.0;
  const size_t nn = (size_t)nb * nb;
  for (int64_t p = inc_ptr[j]; p < inc_ptr[j + 1]; ++p) {
    const int e = inc_cell[p];
    const int l = inc_local[p];
    const uint16_t *sl = slot + (size_t)p * nb;
    const int *ge = gd + (size_t)nb * e;
    // reference-tensor families: 7 weights (tetrahedra) or 4 (triangles)
    constexpr int NT = FAMILY == FFG_TRIANGLE_LAGRANGE ? 4 : 7;
    constexpr bool TENSORS = FAMILY == FFG_TETRA_LAGRANGE || FAMILY == FFG_TRIANGLE_LAGRANGE;
    double gco[NT];
    double F = 0.0;
    if (TENSORS) {
      const double *gg = geo + (size_t)stride * e;
#pragma unroll
      for (int s = 0; s < NT; ++s) gco[s] = gg[s];
      for (int q = 0; q < nq; ++q) F += gg[NT + q] * __ldg(load_basis + (size_t)q * nb + l);
    } else if (FAMILY == FFG_TRIANGLE_P1) {
      F = geo[10 * (size_t)e + 9];
    } else {
      F = cell_rhs[(size_t)nb * e + l];
    }
    for (int i = 0; i < nb; ++i) {
      double kil;
      if (TENSORS) {
        const size_t off = i + (size_t)nb * l;
        kil = 0.0;
#pragma unroll
        for (int s = 0; s < NT; ++s) kil += gco[s] * __ldg(ref + s * nn + off);
      } else if (FAMILY == FFG_TRIANGLE_P1) {
        kil = geo[10 * (size_t)e + i + 3 * l];
      } else if (elem32) {
        kil = (double)elem32[(size_t)cs32 * e + i + (size_t)ld32 * l];
      } else {
        kil = elem[nn * e + i + (size_t)nb * l];
      }
      const uint16_t s = sl[i];
      if (s == kConstrainedSlot) {
        if (g) lift += kil * g[ge[i]];
      } else {
        val64[base + stride_out * s] += kil;
      }
    }
    b += F;
  }
  rhs[out_row] = b - lift;
  if (SELL) {
    double d = 0.0;
    for (int k = 0; k < len; ++k) {
      const double v = val64[base + stride_out * k];
      val32[base + stride_out * k] = (float)v;
      if (row_idx[start + k] == (int)j) d = v;
    }
    const double di = (fabs(d) > 1.0e-14) ? 1.0 / d : 1.0;
    dinv64[out_row] = di;
    dinv32[out_row] = (float)di;
  }
}

template <int FAMILY, bool SELL>
__global__ void column_kernel(int64_t n_free, const int64_t *__restrict__ col_ptr,
                              const int *__restrict__ row_idx, const int64_t *__restrict__ inc_ptr,
                              const int *__restrict__ inc_cell,
                              const uint8_t *__restrict__ inc_local,
                              const uint16_t *__restrict__ slot, const int *__restrict__ gd,
                              int nb, const double *__restrict__ geo, int stride,
                              const double *__restrict__ ref, const double *__restrict__ load_basis,
                              int nq, const double *__restrict__ elem,
                              const double *__restrict__ cell_rhs, const double *__restrict__ g,
                              const int *__restrict__ iperm, const int64_t *__restrict__ soff,
                              double *__restrict__ val64, float *__restrict__ val32,
                              double *__restrict__ dinv64, float *__restrict__ dinv32,
                              double *__restrict__ rhs, const float *__restrict__ elem32,
                              int ld32, int64_t cs32) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n_free)
    column_body<FAMILY, SELL>(j, col_ptr, row_idx, inc_ptr, inc_cell, inc_local, slot, gd, nb, geo,
                              stride, ref, load_basis, nq, elem, cell_rhs, g, iperm, soff, val64,
                              val32, dinv64, dinv32, rhs, elem32, ld32, cs32);
}

// CSC columns of high-order elements (n_b >= 16), one warp per free column:
// the incidences go in ascending cell order as in column_kernel, and for each
// one the lanes take the element's local rows i (distinct rows land in
// distinct slots), adding into the column held in shared memory, so every
// entry receives its terms in the same order as in column_kernel; the
// element column, the slot row and the finished column are read and written
// contiguously.  The lifting is summed per lane and then across the warp in
// a fixed order.  Shared memory: max_len doubles per warp.
template <int FAMILY>
__global__ void csc_column_warp_kernel(int64_t n_free, int max_len,
                                       const int64_t *__restrict__ col_ptr,
                                       const int64_t *__restrict__ inc_ptr,
                                       const int *__restrict__ inc_cell,
                                       const uint8_t *__restrict__ inc_local,
                                       const uint16_t *__restrict__ slot,
                                       const int *__restrict__ gd, int nb,
                                       const double *__restrict__ geo, int stride,
                                       const double *__restrict__ ref,
                                       const double *__restrict__ load_basis, int nq,
                                       const double *__restrict__ elem,
                                       const double *__restrict__ cell_rhs,
                                       const double *__restrict__ g, double *__restrict__ val,
                                       double *__restrict__ rhs, const float *__restrict__ elem32,
                                       int ld32, int64_t cs32) {
  extern __shared__ double col_acc[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t j = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  if (j >= n_free) return;
  const int64_t start = col_ptr[j];
  const int len = (int)(col_ptr[j + 1] - start);
  double *A = col_acc + (size_t)warp * max_len;
  for (int k = lane; k < len; k += 32) A[k] = 0.0;
  __syncwarp();
  const size_t nn = (size_t)nb * nb;
  constexpr int NT = FAMILY == FFG_TRIANGLE_LAGRANGE ? 4 : 7;
  constexpr bool TENSORS = FAMILY == FFG_TETRA_LAGRANGE || FAMILY == FFG_TRIANGLE_LAGRANGE;
  double b = 0.0, lift = 0.0;
  for (int64_t p = inc_ptr[j]; p < inc_ptr[j + 1]; ++p) {
    const int e = inc_cell[p];
    const int l = inc_local[p];
    const uint16_t *sl = slot + (size_t)p * nb;
    const int *ge = gd + (size_t)nb * e;
    double gco[NT];
    double F = 0.0;
    if (TENSORS) {
      const double *gg = geo + (size_t)stride * e;
#pragma unroll
      for (int t = 0; t < NT; ++t) gco[t] = gg[t];
      for (int q = 0; q < nq; ++q) F += gg[NT + q] * __ldg(load_basis + (size_t)q * nb + l);
    } else {
      F = cell_rhs[(size_t)nb * e + l];
    }
    for (int i = lane; i < nb; i += 32) {
      double kil;
      if (TENSORS) {
        const size_t off = i + (size_t)nb * l;
        kil = 0.0;
#pragma unroll
        for (int t = 0; t < NT; ++t) kil += gco[t] * __ldg(ref + t * nn + off);
      } else if (elem32) {
        kil = (double)elem32[(size_t)cs32 * e + i + (size_t)ld32 * l];
      } else {
        kil = elem[nn * e + i + (size_t)nb * l];
      }
      const uint16_t sidx = sl[i];
      if (sidx == kConstrainedSlot) {
        if (g) lift += kil * g[ge[i]];
      } else {
        A[sidx] += kil;
      }
    }
    b += F;
    __syncwarp();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lift += __shfl_xor_sync(0xffffffffu, lift, o);
  for (int k = lane; k < len; k += 32) val[start + k] = A[k];
  if (lane == 0) rhs[j] = b - lift;
}

// SELL rows, one part of a slice (R rows) at a time in CTAs that stay on their
// SM: LR lanes gather one row (free column j = perm[row]) over the element's
// local rows i, as csc_column_warp_kernel does for a CSC column, into the
// part's image in shared memory (slot s of row r at s * (R + 1) + r), every
// entry receiving its terms in ascending incidence order as in column_kernel;
// then the CTA writes the part's FP64 and FP32 values (R * 8 contiguous bytes
// of FP64 per slot step) and clears the image behind it.  Bound: it moves the
// element matrices (Nedelec; the other families' entries are made here), the
// slots and the rows once, and came to issue slots and load latency first, so
// there is one instruction stream for 32 / LR rows, no branch per entry, and
// what the next part needs is loaded a part ahead.
//
// Nedelec (3.2 GB at order 3 on a 24^3 box, 0.5 ms of copy bandwidth), a warp
// per row with a branch per entry and CTAs of one part against this: order 3
// on 24^3 1096 against 693 us, order 4 (FP32 element matrices) on 17 x 16 x 17
// 940 against 693 us; order 6 on 12^3, which went a thread per column, 5406
// against 2212 us.  The other families, a thread per column with read-modify-
// write through L2 (column_kernel) against this: P1 triangles on 64^2 8.5
// against 4.7 us, P2 tetrahedra on 10^3, 21^3 and 48^3 91, 157 and 1197
// against 21, 66 and 613 us, P3 on 14^3 791 against 356 us, Nedelec order 1
// on 15^3 28 against 8 us, five P2 systems of 8^3 to 14^3 in one batch 154
// against 47 us.  The tensor families are bound by L1 wavefronts of the
// reference tensors: 7 NI loads of 32 / LR short segments per incidence step.
struct SliceArgs {
  const int2 *range;  // per SELL row: [p0, p1) of its column's incidences
  int nb, ld32, max_width;
  int64_t cs32;  // FP32 element matrices: elements per cell
  int64_t n_free, n_parts;  // rows, parts of all slices
  const int64_t *soff;
  const int *inc_cell, *gd;
  const uint8_t *inc_local;
  const uint16_t *slot;
  const double *elem, *cell_rhs, *g;
  const double *geo, *ref, *load_basis;  // tensor families and triangles (column_body)
  int stride, nq;
  const float *elem32;
  double *val64, *dinv64, *rhs;
  float *val32, *dinv32;
};
// Threads of a CTA whose groups of LR lanes take one row each: parts of 8, 16
// or 32 rows.
__host__ __device__ constexpr int slice_threads(int lr) { return lr == 4 ? 128 : 256; }

// One row: its incidence range [p0, p1) (empty past the last row) and its
// first LR incidences' cells and local indices, one per lane of its group.
struct SliceRowHead {
  int p0, p1, e, l;
};

__device__ __forceinline__ int2 slice_range(const SliceArgs &A, int64_t row) {
  return row < A.n_free ? A.range[row] : make_int2(0, 0);
}
__device__ __forceinline__ int2 slice_range(const AsmSys &A, int64_t row) {
  if (row >= A.n_free) return make_int2(0, 0);
  const int j = A.perm[row];
  return make_int2((int)A.inc_ptr[j], (int)A.inc_ptr[j + 1]);
}

template <class Args>
__device__ __forceinline__ SliceRowHead slice_head(const Args &A, int2 rg, int i0) {
  SliceRowHead h{rg.x, rg.y, 0, 0};
  if (i0 < rg.y - rg.x) {
    h.e = A.inc_cell[(int64_t)rg.x + i0];
    h.l = A.inc_local[(int64_t)rg.x + i0];
  }
  return h;
}

// The load of local DoF l of cell e (as column_body sums it).
template <int FAMILY, class Args>
__device__ __forceinline__ double slice_load(const Args &A, int e, int l) {
  if constexpr (FAMILY == FFG_TETRA_NEDELEC) {
    return A.cell_rhs[(size_t)A.nb * e + l];
  } else if constexpr (FAMILY == FFG_TRIANGLE_P1) {
    return A.geo[10 * (size_t)e + 9];
  } else {
    const double *gg = A.geo + (size_t)A.stride * e + 7;
    double F = 0.0;
    for (int q = 0; q < A.nq; ++q) F += gg[q] * __ldg(A.load_basis + (size_t)q * A.nb + l);
    return F;
  }
}

// Row r of the part by the calling group of LR lanes (32 / LR rows per warp
// side by side); the lane's local rows are i0, i0 + LR, ..., of which only the
// last can be past nb.  Loads of U incidences are issued before any is added.
// Constrained local rows are added to a slot behind the image that nothing
// reads, so that the adds have no branches.
template <int FAMILY, int NI, int U, bool F32, int LR, class Args>
__device__ __forceinline__ void slice_row(const Args &A, double *img, int r, int64_t row, int i0,
                                          const SliceRowHead &h) {
  constexpr int kPitch = slice_threads(LR) / LR + 1;
  constexpr unsigned kAll = 0xffffffffu;
  const int nb = A.nb;
  const bool tail = i0 + LR * (NI - 1) < nb;
  double b = 0.0, lift = 0.0;
  const int cnt = h.p1 - h.p0;
  const int all = LR == 32 ? cnt : __reduce_max_sync(kAll, cnt);
  int dslot = A.max_width;
  for (int base = 0; base < all; base += LR) {
    int e = h.e, l = h.l;
    if (base > 0) {
      const int64_t p = (int64_t)h.p0 + base + i0;
      e = base + i0 < cnt ? A.inc_cell[p] : 0;
      l = base + i0 < cnt ? A.inc_local[p] : 0;
    }
    // the lane's incidence: the offset of its element column and its load
    size_t my_col = 0;
    if constexpr (FAMILY == FFG_TETRA_NEDELEC)
      my_col = F32 ? (size_t)e * (size_t)A.cs32 + (size_t)(A.ld32 * l)
                   : ((size_t)e * nb + l) * (size_t)nb;
    else if constexpr (FAMILY == FFG_TRIANGLE_P1)
      my_col = 10 * (size_t)e + 3 * l;
    const double my_f = base + i0 < cnt ? slice_load<FAMILY>(A, e, l) : 0.0;
    const uint16_t *slp = A.slot + ((size_t)h.p0 + base) * nb + i0;
    const int n = min(LR, all - base);
    for (int u0 = 0; u0 < n; u0 += U) {
      double kil[U][NI];
      int sl[U][NI];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool live = base + u0 + u < cnt;
        const int from = (u0 + u) & (LR - 1);
#pragma unroll
        for (int c = 0; c < NI; ++c)
          sl[u][c] = live && (c < NI - 1 || tail) ? (int)__ldg(slp + LR * c)
                                                  : (int)kConstrainedSlot;
        if constexpr (FAMILY == FFG_TETRA_LAGRANGE) {
          const double *gg = A.geo + (size_t)A.stride * __shfl_sync(kAll, e, from, LR);
          const double *rf = A.ref + nb * __shfl_sync(kAll, l, from, LR) + i0;
          double gco[7];
#pragma unroll
          for (int t = 0; t < 7; ++t) gco[t] = __ldg(gg + t);
#pragma unroll
          for (int c = 0; c < NI; ++c) {
            kil[u][c] = 0.0;
            if (c < NI - 1 || tail) {
#pragma unroll
              for (int t = 0; t < 7; ++t)
                kil[u][c] += gco[t] * __ldg(rf + t * nb * nb + LR * c);
            }
          }
        } else {
          const size_t col = __shfl_sync(kAll, my_col, from, LR) + i0;
#pragma unroll
          for (int c = 0; c < NI; ++c) {
            const bool in = live && (c < NI - 1 || tail);
            if constexpr (FAMILY == FFG_TRIANGLE_P1)
              kil[u][c] = in ? __ldg(A.geo + col + LR * c) : 0.0;
            else if constexpr (F32)
              kil[u][c] = in ? (double)__ldg(A.elem32 + col + LR * c) : 0.0;
            else
              kil[u][c] = in ? __ldg(A.elem + col + LR * c) : 0.0;
          }
        }
        slp += nb;
      }
      // the diagonal's slot: local row l of any incidence (e, l) of column j
      // has global DoF j, so its slot entry is the diagonal
      if (u0 == 0 && base == 0) {
        const int l0 = __shfl_sync(kAll, l, 0, LR);
#pragma unroll
        for (int c = 0; c < NI; ++c)
          if (i0 + LR * c == l0) dslot = sl[0][c];
        dslot = min(__shfl_sync(kAll, dslot, l0 & (LR - 1), LR), A.max_width);
      }
      if (A.g) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int *ge = A.gd + (size_t)nb * __shfl_sync(kAll, e, (u0 + u) & (LR - 1), LR) + i0;
#pragma unroll
          for (int c = 0; c < NI; ++c)
            if (sl[u][c] == kConstrainedSlot && base + u0 + u < cnt && (c < NI - 1 || tail))
              lift += kil[u][c] * A.g[ge[LR * c]];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int c = 0; c < NI; ++c)
          img[min(sl[u][c], A.max_width) * kPitch + r] += kil[u][c];
        b += __shfl_sync(kAll, my_f, (u0 + u) & (LR - 1), LR);
        __syncwarp();
      }
    }
  }
  if (A.g) {
#pragma unroll
    for (int o = LR / 2; o > 0; o >>= 1) lift += __shfl_xor_sync(kAll, lift, o);
  }
  if (i0 == 0 && row < A.n_free) {
    const double d = dslot < A.max_width ? img[dslot * kPitch + r] : 0.0;
    const double di = (fabs(d) > 1.0e-14) ? 1.0 / d : 1.0;
    A.dinv64[row] = di;
    A.dinv32[row] = (float)di;
    A.rhs[row] = b - lift;
  }
}

// The part's image to its slice, starting at entry `at`; the image is cleared.
template <int LR, class Args>
__device__ __forceinline__ void slice_write(const Args &A, double *img, int64_t at, int width) {
  constexpr int R = slice_threads(LR) / LR;
  for (int t = threadIdx.x; t < width * (R / 2); t += slice_threads(LR)) {
    const int sl = t / (R / 2), rr = 2 * (t % (R / 2));
    double *p = img + sl * (R + 1) + rr;
    const double2 v = {p[0], p[1]};
    p[0] = 0.0;
    p[1] = 0.0;
    const int64_t o = at + sl * kSliceRows + rr;
    *reinterpret_cast<double2 *>(A.val64 + o) = v;
    *reinterpret_cast<float2 *>(A.val32 + o) = make_float2((float)v.x, (float)v.y);
  }
}

// The next part's incidences and the ranges of the one after it are loaded
// while a part is gathered, so that the chain range -> incidence -> element
// column costs one memory latency per part.
template <int FAMILY, int NI, int U, bool F32, int LR, int CTAS>
__global__ void __launch_bounds__(slice_threads(LR), CTAS)
sell_slice_kernel(const __grid_constant__ SliceArgs A) {
  extern __shared__ double img[];
  constexpr int R = slice_threads(LR) / LR, kParts = kSliceRows / R;
  const int r = threadIdx.x / LR, i0 = threadIdx.x % LR;
  const int64_t step = gridDim.x;
  SliceRowHead h = slice_head(A, slice_range(A, blockIdx.x * (int64_t)R + r), i0);
  int2 rg = slice_range(A, (blockIdx.x + step) * R + r);
  for (int q = threadIdx.x; q < (A.max_width + 1) * (R + 1); q += slice_threads(LR)) img[q] = 0.0;
  __syncthreads();
  for (int64_t part = blockIdx.x; part < A.n_parts; part += step) {
    const int64_t row = part * R + r;
    const int64_t s0 = A.soff[part / kParts], s1 = A.soff[part / kParts + 1];
    const SliceRowHead hn = slice_head(A, rg, i0);
    rg = slice_range(A, row + 2 * step * R);
    slice_row<FAMILY, NI, U, F32, LR>(A, img, r, row, i0, h);
    __syncthreads();
    slice_write<LR>(A, img, s0 + (part % kParts) * R, (int)((s1 - s0) / kSliceRows));
    __syncthreads();
    h = hn;
  }
}

inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }

// ------------------------------------------- batched assembly (serving)
// Independent systems of one family assembled by one launch per phase: a
// thread finds its system by binary search over the prefix sums of cells
// (geometry) or free columns (scatter) and runs the same per-cell / per-column
// body as the single-system kernels, so every system's values are the bits
// it gets alone.
__device__ __forceinline__ int batch_find(const int64_t *begin, int count, int64_t g) {
  int lo = 0, hi = count;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (begin[mid] <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

__global__ void batch_prep_kernel(const __grid_constant__ AsmBatch B) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < B.count) *B.sys[s].err = 0;
}

template <int FAMILY>
__global__ void batch_geometry_kernel(const __grid_constant__ AsmBatch B) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= B.cell_begin[B.count]) return;
  const int s = batch_find(B.cell_begin, B.count, g);
  const AsmSys &S = B.sys[s];
  const int c = (int)(g - B.cell_begin[s]);
  if (FAMILY == FFG_TETRA_LAGRANGE)
    lagrange_geometry_cell(c, S.cells, S.verts, S.ca, S.cb, S.cell_a, S.cell_b, S.samples, S.nq,
                           S.geo, S.stride, S.err);
  else
    p1_geometry_cell(c, S.cells, S.verts, S.ca, S.cb, S.cell_a, S.cell_b, S.samples, S.geo, S.err);
}

// The parts of every system's slices, one per CTA, and x = 0 for its solve.
template <int FAMILY, int NI, int LR>
__global__ void __launch_bounds__(slice_threads(LR))
batch_slice_kernel(const __grid_constant__ AsmBatch B) {
  extern __shared__ double img[];
  constexpr int R = slice_threads(LR) / LR, kParts = kSliceRows / R;
  const int s = batch_find(B.col_begin, B.count, blockIdx.x);
  const AsmSys &S = B.sys[s];
  const int64_t part = blockIdx.x - B.col_begin[s];
  const int r = threadIdx.x / LR, i0 = threadIdx.x % LR;
  const int64_t row = part * R + r;
  const SliceRowHead h = slice_head(S, slice_range(S, row), i0);
  const int64_t s0 = S.soff[part / kParts], s1 = S.soff[part / kParts + 1];
  for (int q = threadIdx.x; q < (S.max_width + 1) * (R + 1); q += slice_threads(LR)) img[q] = 0.0;
  if (i0 == 0 && row < S.n_free) S.x[row] = 0.0;
  __syncthreads();
  slice_row<FAMILY, NI, 1, false, LR>(S, img, r, row, i0, h);
  __syncthreads();
  slice_write<LR>(S, img, s0 + (part % kParts) * R, (int)((s1 - s0) / kSliceRows));
}

// the SELL-layout scatter of every system, and x = 0 for its solve
template <int FAMILY>
__global__ void batch_column_kernel(const __grid_constant__ AsmBatch B) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= B.col_begin[B.count]) return;
  const int s = batch_find(B.col_begin, B.count, g);
  const AsmSys &S = B.sys[s];
  const int64_t j = g - B.col_begin[s];
  S.x[j] = 0.0;
  column_body<FAMILY, true>(j, S.col_ptr, S.row_idx, S.inc_ptr, S.inc_cell, S.inc_local, S.slot,
                            S.gd, S.nb, S.geo, S.stride, S.ref, S.load_basis, S.nq, nullptr,
                            nullptr, S.g, S.iperm, S.soff, S.val64, S.val32, S.dinv64, S.dinv32,
                            S.rhs, nullptr, 0, 0);
}

// every system's full solution: constrained DoFs from g (or 0), free DoFs
// from the solver's x (SELL order)
__global__ void batch_solution_kernel(const __grid_constant__ AsmBatch B) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= B.dof_begin[B.count]) return;
  const int s = batch_find(B.dof_begin, B.count, g);
  const AsmSys &S = B.sys[s];
  const int64_t d = g - B.dof_begin[s];
  const int f = S.free_index[d];
  S.solution[d] = f >= 0 ? S.x[S.iperm[f]] : (S.g ? S.g[d] : 0.0);
}

}  // namespace

namespace {

constexpr size_t kSliceImage = 224 * 1024;  // image bytes of an SM's CTAs

// Lanes per row of the slice gather, 0 where a part's image does not fit on an
// SM.  Narrow groups keep their lanes full on small elements and share one
// instruction stream between more rows, but have more rows per image: the
// narrowest for which three images fit on an SM, else a warp per row (16 lanes
// for the tensor families) while one does.
int slice_lanes(int family, int nb, int64_t max_column) {
  auto image = [&](int lr) {
    return sizeof(double) * (size_t)(max_column + 1) * (slice_threads(lr) / lr + 1);
  };
  if (max_column <= 0) return 0;
  int first = 32, last = 32;
  if (family == FFG_TETRA_NEDELEC) {
    first = nb < 16 ? 8 : nb <= 96 ? 16 : 32;
    last = nb < 16 ? 8 : 32;
  } else if (family == FFG_TRIANGLE_P1) {
    first = last = 4;
  } else if (family == FFG_TETRA_LAGRANGE) {
    first = nb == 4 ? 4 : 8;
    last = nb == 4 ? 4 : 16;
  } else {
    return 0;
  }
  if (image(first) <= kSliceImage / 3) return first;
  return image(last) <= kSliceImage ? last : 0;
}
size_t slice_bytes(int lr, int64_t max_column) {
  return sizeof(double) * (size_t)(max_column + 1) * (slice_threads(lr) / lr + 1);
}

// Opts a kernel into the largest image.  Always into the same size: another
// thread may be between this and its launch of the same kernel for another mesh.
template <class Kernel>
bool allow_images(Kernel kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kSliceImage) == cudaSuccess;
}

template <int FAMILY, bool F32>
int launch_slices(const SliceArgs &A, int lanes, size_t smem, cudaStream_t s) {
  auto go = [&](auto kern) -> int {
    const int threads = slice_threads(lanes);
    int dev = 0, sms = 0, ctas = 0;
    if (!allow_images(kern) || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kern, threads, smem) !=
            cudaSuccess ||
        ctas < 1)
      return FFG_CUDA_ERROR;
    const int64_t grid = std::min<int64_t>(A.n_parts, (int64_t)sms * ctas);
    kern<<<(unsigned)grid, threads, smem, s>>>(A);
    return cudaGetLastError() == cudaSuccess ? FFG_OK : FFG_CUDA_ERROR;
  };
  const int ni = (A.nb + lanes - 1) / lanes;
  if constexpr (FAMILY == FFG_TETRA_NEDELEC) {
    // U and the CTAs per SM (the registers) by timing orders 3, 4 and 6: more
    // loads in flight per warp at fewer warps, or fewer at spilled registers,
    // both measured 5 % to 40 % slower
    if (lanes == 8) return go(sell_slice_kernel<FAMILY, 1, 2, F32, 8, 4>);
    if (lanes == 16) {
      if (ni == 2) return go(sell_slice_kernel<FAMILY, 2, 2, F32, 16, 4>);
      if (ni == 3) return go(sell_slice_kernel<FAMILY, 3, 1, F32, 16, 5>);
      if (ni == 6) return go(sell_slice_kernel<FAMILY, 6, 1, F32, 16, 4>);
    } else {
      if (ni == 1) return go(sell_slice_kernel<FAMILY, 1, 1, F32, 32, 4>);
      if (ni == 2) return go(sell_slice_kernel<FAMILY, 2, 1, F32, 32, 4>);
      if (ni == 3) return go(sell_slice_kernel<FAMILY, 3, 1, F32, 32, 4>);
      if (ni == 5) return go(sell_slice_kernel<FAMILY, 5, 1, F32, 32, 4>);
      if (ni == 7) return go(sell_slice_kernel<FAMILY, 7, 1, F32, 32, 3>);
    }
  } else if constexpr (FAMILY == FFG_TRIANGLE_P1) {
    return go(sell_slice_kernel<FAMILY, 1, 1, false, 4, 8>);
  } else {
    if (lanes == 4) return go(sell_slice_kernel<FAMILY, 1, 1, false, 4, 8>);
    if (lanes == 8) {
      if (ni == 2) return go(sell_slice_kernel<FAMILY, 2, 1, false, 8, 4>);
      if (ni == 3) return go(sell_slice_kernel<FAMILY, 3, 1, false, 8, 4>);
      if (ni == 5) return go(sell_slice_kernel<FAMILY, 5, 1, false, 8, 4>);
    } else {
      if (ni == 1) return go(sell_slice_kernel<FAMILY, 1, 1, false, 16, 4>);
      if (ni == 2) return go(sell_slice_kernel<FAMILY, 2, 1, false, 16, 4>);
      if (ni == 3) return go(sell_slice_kernel<FAMILY, 3, 1, false, 16, 4>);
    }
  }
  return FFG_INVALID_INPUT;
}

// The slices of the batch's systems, all of one nb and one lane count.
int launch_batch_slices(int family, int lanes, AsmBatch &B, cudaStream_t s) {
  const int rows = slice_threads(lanes) / lanes;
  int max_width = 0;
  for (int i = 0; i < B.count; ++i) {
    max_width = std::max(max_width, B.sys[i].max_width);
    B.col_begin[i + 1] = B.col_begin[i] + (B.sys[i].n_free + kSliceRows - 1) / kSliceRows *
                                              (kSliceRows / rows);
  }
  const int64_t parts = B.col_begin[B.count];
  if (!parts) return FFG_OK;
  const size_t smem = slice_bytes(lanes, max_width);
  auto go = [&](auto kern) -> int {
    if (!allow_images(kern)) return FFG_CUDA_ERROR;
    kern<<<(unsigned)parts, slice_threads(lanes), smem, s>>>(B);
    return cudaGetLastError() == cudaSuccess ? FFG_OK : FFG_CUDA_ERROR;
  };
  if (family == FFG_TRIANGLE_P1) return go(batch_slice_kernel<FFG_TRIANGLE_P1, 1, 4>);
  const int ni = (B.sys[0].nb + lanes - 1) / lanes;
  if (lanes == 4) return go(batch_slice_kernel<FFG_TETRA_LAGRANGE, 1, 4>);
  if (lanes == 8) {
    if (ni == 2) return go(batch_slice_kernel<FFG_TETRA_LAGRANGE, 2, 8>);
    if (ni == 3) return go(batch_slice_kernel<FFG_TETRA_LAGRANGE, 3, 8>);
    if (ni == 5) return go(batch_slice_kernel<FFG_TETRA_LAGRANGE, 5, 8>);
  } else {
    if (ni == 1) return go(batch_slice_kernel<FFG_TETRA_LAGRANGE, 1, 16>);
    if (ni == 2) return go(batch_slice_kernel<FFG_TETRA_LAGRANGE, 2, 16>);
    if (ni == 3) return go(batch_slice_kernel<FFG_TETRA_LAGRANGE, 3, 16>);
  }
  return FFG_INVALID_INPUT;
}

}  // namespace

int launch_batch_assembly(int family, int count, const AsmSys *sys, cudaStream_t s) {
  if (family != FFG_TETRA_LAGRANGE && family != FFG_TRIANGLE_P1) return FFG_INVALID_INPUT;
  // one launch per phase for the systems of one element size and lane count
  // (a system is gathered here as it is alone)
  std::vector<int> left(count);
  for (int i = 0; i < count; ++i) left[i] = i;
  auto lanes_of = [&](int i) { return slice_lanes(family, sys[i].nb, sys[i].max_width); };
  while (!left.empty()) {
    const int nb = sys[left[0]].nb, lanes = lanes_of(left[0]);
    AsmBatch B;
    B.count = 0;
    B.cell_begin[0] = B.col_begin[0] = B.dof_begin[0] = 0;
    std::vector<int> rest;
    for (int i : left) {
      if (sys[i].nb != nb || lanes_of(i) != lanes || B.count == kMaxAsmBatch) {
        rest.push_back(i);
        continue;
      }
      const int k = B.count++;
      B.sys[k] = sys[i];
      B.cell_begin[k + 1] = B.cell_begin[k] + sys[i].n_cells;
      B.col_begin[k + 1] = B.col_begin[k] + sys[i].n_free;
      B.dof_begin[k + 1] = B.dof_begin[k] + sys[i].n_dofs;
    }
    left.swap(rest);
    batch_prep_kernel<<<1, kMaxAsmBatch, 0, s>>>(B);
    const int64_t nc = B.cell_begin[B.count], nf = B.col_begin[B.count];
    if (family == FFG_TETRA_LAGRANGE) {
      if (nc) batch_geometry_kernel<FFG_TETRA_LAGRANGE><<<blocks_for(nc, 128), 128, 0, s>>>(B);
      if (nf && !lanes)
        batch_column_kernel<FFG_TETRA_LAGRANGE><<<blocks_for(nf, 128), 128, 0, s>>>(B);
    } else {
      if (nc) batch_geometry_kernel<FFG_TRIANGLE_P1><<<blocks_for(nc, 128), 128, 0, s>>>(B);
      if (nf && !lanes)
        batch_column_kernel<FFG_TRIANGLE_P1><<<blocks_for(nf, 128), 128, 0, s>>>(B);
    }
    if (cudaGetLastError() != cudaSuccess) return FFG_CUDA_ERROR;
    if (lanes) {
      if (int st = launch_batch_slices(family, lanes, B, s)) return st;
    }
  }
  return FFG_OK;
}

int launch_batch_solutions(int count, const AsmSys *sys, cudaStream_t s) {
  for (int c0 = 0; c0 < count; c0 += kMaxAsmBatch) {
    AsmBatch B;
    B.count = std::min(kMaxAsmBatch, count - c0);
    B.dof_begin[0] = 0;
    for (int i = 0; i < B.count; ++i) {
      B.sys[i] = sys[c0 + i];
      B.dof_begin[i + 1] = B.dof_begin[i] + B.sys[i].n_dofs;
    }
    const int64_t nd = B.dof_begin[B.count];
    if (nd) batch_solution_kernel<<<blocks_for(nd, 256), 256, 0, s>>>(B);
    if (cudaGetLastError() != cudaSuccess) return FFG_CUDA_ERROR;
  }
  return FFG_OK;
}

int launch_cell_geometry(const Topology &t, const ElementTables &tab, const DeviceTopology &dt,
                         const AssemblyInputs &in, double *geo, int stride, double *cell_rhs,
                         int *err, cudaStream_t s) {
  (void)cell_rhs;
  const int T = 128;
  if (t.family == FFG_TETRA_LAGRANGE) {
    lagrange_geometry_kernel<<<blocks_for(t.n_cells, T), T, 0, s>>>(
        t.n_cells, dt.cells, in.vertices, in.coef_a, in.coef_b, in.cell_a, in.cell_b, in.samples,
        tab.nq_load, geo, stride, err);
  } else if (t.family == FFG_TRIANGLE_LAGRANGE) {
    triangle_lagrange_geometry_kernel<<<blocks_for(t.n_cells, T), T, 0, s>>>(
        t.n_cells, dt.cells, in.vertices, in.coef_a, in.coef_b, in.cell_a, in.cell_b, in.samples,
        tab.nq_load, geo, stride, err);
  } else if (t.family == FFG_TRIANGLE_P1) {
    p1_geometry_kernel<<<blocks_for(t.n_cells, T), T, 0, s>>>(t.n_cells, dt.cells, in.vertices,
                                                             in.coef_a, in.coef_b, in.cell_a,
                                                             in.cell_b, in.samples, geo, err);
  }
  return cudaGetLastError() == cudaSuccess ? FFG_OK : FFG_CUDA_ERROR;
}

int launch_nedelec(const Topology &t, const ElementTables &tab, const DeviceTopology &dt,
                   const AssemblyInputs &in, double *elem, double *cell_rhs, int *err,
                   cudaStream_t s, bool load_only) {
  (void)tab;
  if (!dt.ort) return FFG_INVALID_INPUT;
  return launch_nedelec_oriented(t, *dt.ort, dt, in, elem, cell_rhs, err, s, load_only);
}

namespace {
int sell_slice_lanes(const Topology &t, const DeviceSell &sell) {
  return sell.inc_range ? slice_lanes(t.family, t.nb, t.max_column) : 0;
}
}  // namespace

bool sell_by_slices(const Topology &t, const DeviceSell &sell) {
  return sell_slice_lanes(t, sell) != 0;
}

int launch_columns(const Topology &t, const ElementTables &tab, const DeviceTopology &dt,
                   const AssemblyInputs &in, const double *geo, int stride,
                   const double *cell_rhs, const double *elem, const int64_t *col_ptr,
                   const int *row_idx, DeviceSell *sell, double *csc_val, double *rhs,
                   cudaStream_t s, const float *elem32, int ld32, int64_t cs32) {
  if (elem32 && cs32 <= 0) cs32 = (int64_t)ld32 * t.nb;
  const int T = (in.tune && in.tune->col_threads) ? in.tune->col_threads : 128;
  const int64_t F = t.n_free();
  if (F == 0) return FFG_OK;
  const int *iperm = sell ? sell->iperm : nullptr;
  const int64_t *soff = sell ? sell->soff : nullptr;
  double *v64 = sell ? sell->val64 : csc_val;
  float *v32 = sell ? sell->val32 : nullptr;
  double *d64 = sell ? sell->dinv64 : nullptr;
  float *d32 = sell ? sell->dinv32 : nullptr;
#define FFG_COLUMN_ARGS                                                                        \
  F, col_ptr, row_idx, dt.inc_ptr, dt.inc_cell, dt.inc_local, dt.slot, dt.gd, t.nb, geo, stride, \
      dt.ref, dt.load_basis, tab.nq_load, elem, cell_rhs, in.g, iperm, soff, v64, v32, d64, d32, rhs, \
      elem32, ld32, cs32
  // high-order CSC columns: one warp per column (48 KB of columns per block)
  constexpr int kColSmem = 48 * 1024;
  const int col_bytes = t.max_column * (int)sizeof(double);
  const bool by_warp = !sell && t.nb >= 16 && t.family != FFG_TRIANGLE_P1 && t.max_column > 0 &&
                       col_bytes <= kColSmem;
  const int wpb = by_warp ? std::max(1, std::min(8, kColSmem / col_bytes)) : 0;
  // SELL rows by the slice gather
  const int lanes = sell ? sell_slice_lanes(t, *sell) : 0;
  if (lanes) {
    SliceArgs A;
    A.range = sell->inc_range;
    A.nb = t.nb;
    A.ld32 = ld32;
    A.max_width = t.max_column;
    A.cs32 = cs32;
    A.n_free = F;
    A.n_parts = sell->n_slices * (kSliceRows * lanes / slice_threads(lanes));
    A.soff = sell->soff;
    A.inc_cell = dt.inc_cell;
    A.gd = dt.gd;
    A.inc_local = dt.inc_local;
    A.slot = dt.slot;
    A.elem = elem;
    A.cell_rhs = cell_rhs;
    A.g = in.g;
    A.geo = geo;
    A.ref = dt.ref;
    A.load_basis = dt.load_basis;
    A.stride = stride;
    A.nq = tab.nq_load;
    A.elem32 = elem32;
    A.val64 = sell->val64;
    A.dinv64 = sell->dinv64;
    A.rhs = rhs;
    A.val32 = sell->val32;
    A.dinv32 = sell->dinv32;
    const size_t smem = slice_bytes(lanes, t.max_column);
    if (t.family == FFG_TETRA_LAGRANGE)
      return launch_slices<FFG_TETRA_LAGRANGE, false>(A, lanes, smem, s);
    if (t.family == FFG_TRIANGLE_P1)
      return launch_slices<FFG_TRIANGLE_P1, false>(A, lanes, smem, s);
    return elem32 ? launch_slices<FFG_TETRA_NEDELEC, true>(A, lanes, smem, s)
                  : launch_slices<FFG_TETRA_NEDELEC, false>(A, lanes, smem, s);
  }
#define FFG_LAUNCH(FAM)                                                                        \
  do {                                                                                         \
    if (sell)                                                                                  \
      column_kernel<FAM, true><<<blocks_for(F, T), T, 0, s>>>(FFG_COLUMN_ARGS);                \
    else if (by_warp && FAM != FFG_TRIANGLE_P1)                                                \
      csc_column_warp_kernel<FAM><<<(unsigned)((F + wpb - 1) / wpb), 32 * wpb,                 \
                                    (size_t)wpb * col_bytes, s>>>(                             \
          F, t.max_column, col_ptr, dt.inc_ptr, dt.inc_cell, dt.inc_local, dt.slot, dt.gd,      \
          t.nb, geo, stride, dt.ref, dt.load_basis, tab.nq_load, elem, cell_rhs, in.g, v64,    \
          rhs, elem32, ld32, cs32);                                                                  \
    else                                                                                       \
      column_kernel<FAM, false><<<blocks_for(F, T), T, 0, s>>>(FFG_COLUMN_ARGS);               \
  } while (0)
  if (t.family == FFG_TETRA_LAGRANGE)
    FFG_LAUNCH(FFG_TETRA_LAGRANGE);
  else if (t.family == FFG_TRIANGLE_P1)
    FFG_LAUNCH(FFG_TRIANGLE_P1);
  else if (t.family == FFG_TRIANGLE_LAGRANGE)
    FFG_LAUNCH(FFG_TRIANGLE_LAGRANGE);
  else
    FFG_LAUNCH(FFG_TETRA_NEDELEC);
#undef FFG_LAUNCH
#undef FFG_COLUMN_ARGS
  return cudaGetLastError() == cudaSuccess ? FFG_OK : FFG_CUDA_ERROR;
}

}  // namespace ffg
