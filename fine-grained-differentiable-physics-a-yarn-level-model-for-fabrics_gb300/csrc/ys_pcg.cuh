// ys_pcg.cuh -- the Jacobi-PCG's device arithmetic, shared by the phase kernels
// (ys_kernels.cu) and the persistent solve (ys_pcg_cluster.cu), so that both
// give the same bits.
//
// A group of 32 consecutive nodes has four warps: warp part m < 3 computes row
// m of the node's x rows, 45 of the row block's 159 coefficients, part 3 the
// two Eulerian rows, 24. An SM issues one warp's FP64 instruction over 64
// cycles of one of its four pipes, so a thread per node left three of them idle
// on small cloths; split by rows every sum keeps its order.
#pragma once

#include "ys_items.cuh"
#include "ys_kernels.cuh"

namespace ys {

constexpr int kGroup = 32;     // nodes of a group
constexpr int kRowCoefs = 45;  // coefficients of an x row; the Eulerian rows have 24

// The PCG's arithmetic, written once for every schedule (the contraction is
// spelled out, so the bits do not depend on what the compiler fuses).
// z = D^-1 r of one component, and its terms of |r|^2 and r.z
__device__ __forceinline__ double pcg_norms(double r, double dinv, double& rr, double& rz) {
  const double z = dinv * r;
  rr = fma(r, r, rr);
  rz = fma(r, z, rz);
  return z;
}
// the step along p
__device__ __forceinline__ void pcg_advance(double alpha, double p, double q, double& x, double& r) {
  x = fma(alpha, p, x);
  r = fma(-alpha, q, r);
}
__device__ __forceinline__ double pcg_threshold(double tol, double bb) {
  const double thr = tol * tol * bb;
  return thr < 2.2250738585072014e-308 ? 2.2250738585072014e-308 : thr;
}
// Coefficient j of row part m of row block n of A, or of A^T (TRANS: read from
// the rows of the neighbours, 0 where there is none), in the order of
// spmv_row_sv and spmv_row_tv. i(du, dv): the row to read for the neighbour
// there, negative outside the cloth.
template <bool TRANS, class Row>
__device__ __forceinline__ double row_coef(const double* A, int64_t nt, int n, int m, int j,
                                           const Row& i) {
  auto at = [&](int slot, int row) { return row < 0 ? 0.0 : A[(int64_t)slot * nt + row]; };
  auto nbr = [&](int mm) { return TRANS ? i(mm == 0 ? -1 : mm == 1 ? 1 : 0, mm == 2 ? -1 : mm == 3 ? 1 : 0) : n; };
  if (m < 3) {
    if (j < 39) {
      const int s = j / 3, c = j - 3 * s;
      return at(YS_SLOT_LL + 9 * s + (TRANS ? 3 * c + m : 3 * m + c), TRANS ? i(stencil_du(s), stencil_dv(s)) : n);
    }
    if (j < 41) return at(TRANS ? YS_SLOT_EL_SELF + 3 * (j - 39) + m : YS_SLOT_LE_SELF + 2 * m + (j - 39), n);
    return at((TRANS ? YS_SLOT_EL_NBR : YS_SLOT_LE_NBR) + 3 * (j - 41) + m, nbr(j - 41));
  }
  const int k = j / 12, e = j - 12 * k;
  if (e < 3) return at(TRANS ? YS_SLOT_LE_SELF + 2 * e + k : YS_SLOT_EL_SELF + 3 * k + e, n);
  if (e == 3) return at(YS_SLOT_EE_SELF + k, n);
  const int mm = 2 * k + (e >= 8), c = (e - 4) & 3;
  if (c < 3) return at((TRANS ? YS_SLOT_LE_NBR : YS_SLOT_EL_NBR) + 3 * mm + c, nbr(mm));
  return at(YS_SLOT_EE_NBR + mm, nbr(mm));
}

// y = the rows of part m times x: y[0] of x row m, y[0..1] of the two Eulerian
// rows. coef(j): row_coef's; x(c, du, dv): component c of the neighbour there,
// any finite number outside the cloth (the coefficient is 0).
template <bool TRANS, class Coef, class Vec>
__device__ __forceinline__ void row_product(int m, const Coef& coef, const Vec& x, double y[2]) {
  constexpr int sg = TRANS ? -1 : 1;
  if (m < 3) {
    double s = 0.0;
#pragma unroll
    for (int t = 0; t < kNumStencil; ++t) {
#pragma unroll
      for (int c = 0; c < 3; ++c) s = fma(coef(3 * t + c), x(c, sg * stencil_du(t), sg * stencil_dv(t)), s);
    }
    s = fma(coef(39), x(3, 0, 0), s);
    s = fma(coef(40), x(4, 0, 0), s);
    s = fma(coef(41), x(3, -sg, 0), s);
    s = fma(coef(42), x(3, sg, 0), s);
    s = fma(coef(43), x(4, 0, -sg), s);
    s = fma(coef(44), x(4, 0, sg), s);
    y[0] = s;
    y[1] = 0.0;
  } else {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int du = k == 0 ? sg : 0, dv = k == 0 ? 0 : sg, b = 12 * k;
      double e = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) e = fma(coef(b + c), x(c, 0, 0), e);
      e = fma(coef(b + 3), x(3 + k, 0, 0), e);
#pragma unroll
      for (int c = 0; c < 3; ++c) e = fma(coef(b + 4 + c), x(c, -du, -dv), e);
      e = fma(coef(b + 7), x(3 + k, -du, -dv), e);
#pragma unroll
      for (int c = 0; c < 3; ++c) e = fma(coef(b + 8 + c), x(c, du, dv), e);
      e = fma(coef(b + 11), x(3 + k, du, dv), e);
      y[k] = e;
    }
  }
}

// four group sums of a block; n lanes' sums (zero elsewhere): the levels of the
// tree that would add zeros are left out
__device__ __forceinline__ double four_sum(double a, double b, double c, double d) { return (a + b) + (c + d); }
__device__ __forceinline__ double lanes_sum(double s, int n) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < n) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// fixed-order sum of cloth c's block partials in row `which`, by a whole warp:
// lane l adds blocks l, l + 32, ... in order, then the lanes as a tree. (One
// thread adding them all waited out an FP64 addition per block, up to 79 of
// them on a 100 x 100 cloth, in every block of every launch.)
__device__ __forceinline__ double cloth_sum(const Blocks& b, const double* part, int which, int c) {
  const int b0 = b.cloth_blk0[c], nb = b.cloth_nblk[c];
  double s = 0.0;
  for (int i = threadIdx.x & 31; i < nb; i += 32) s += part[which * b.nblk + b0 + i];
  return lanes_sum(s, nb);
}

// where the groups' p.q partials start in Solver::part
__device__ __forceinline__ int64_t pq_row(const Blocks& b) { return 4LL * b.nblk; }
// the sum of p.q: its partials are kept per block (row 0), or per group of 32
// nodes (by_rows), four to a block
__device__ __forceinline__ double cloth_sum_pq(const Blocks& b, const double* part, int c) {
  if (!b.by_rows) return cloth_sum(b, part, 0, c);
  const int b0 = b.cloth_blk0[c], nb = b.cloth_nblk[c];
  double s = 0.0;
  for (int i = threadIdx.x & 31; i < nb; i += 32) {
    const double* g = part + pq_row(b) + 4LL * (b0 + i);
    s += four_sum(g[0], g[1], g[2], g[3]);
  }
  return lanes_sum(s, nb);
}

}  // namespace ys
