// ys_adjoint.cu -- kernels of the reverse-mode (adjoint) step.
//
// One step maps the state s = (LPos, LVel, EPos, EVel, EPosBar) and the
// parameters to s' through: assembly of A(s), b(s); q = A^-1 b; Cloth::update
// (src/Cloth.cpp:111-148). Given the adjoint g' = dL/ds', the adjoint step
// returns dL/ds, dL/d(parameters) and dL/d(external force):
//
//   1. the update's transpose: q_bar from g' (k_adj_update), the slide
//      indicator's adjoint, and the parts of g' that pass straight through;
//   2. lambda = A^-T q_bar (exact), or A^-1 q_bar (the reference's own
//      backward of its solve, src/Solvers.cpp:33-58), by the PCG kernels;
//   3. the gradient of phi = lambda . (b(s) - A(s) q) + slide_bar . slide(s)
//      (without A q in the reference mode, whose A carries no graph), q and
//      lambda held fixed.
//
// phi is a sum over elements: each edge, bend segment, face and shear segment
// gives its record's fields times fixed weights (products of lambda and q at
// its nodes), so its gradient with respect to its own few inputs (15 of an
// edge, 8 and 7 of a bend segment, 9 of a face, 7 of a shear segment) is taken
// by evaluating the element code (ys_physics.cuh) over Dual<2>, a pair of
// inputs per thread, and no record is stored. The terms that couple elements
// are undone by hand in reverse order: shear needs the crossing's compression,
// friction the gathered force and crimp sums, crimp bending the normals.
//
//   k_adj_shear     d phi / d(arms, (compression + 1) S R^2) per segment
//   k_adj_cross     friction: adjoints of the gathered forces and crimp sums,
//                   of the normal, EPos, EPosBar, EVel, mu per crossing
//   k_adj_edge, k_adj_bend, k_adj_face   per element, with those adjoints
//   k_adj_normal    normal -> positions of its five crossings
//   k_adj_gather    per node, in a fixed order, no atomics
//   k_adj_params    per yarn line and cloth
//
// Bound by the FP64 pipe on large cloths and by latency on small ones: about
// 90,000 FP64 operations a node. Two inputs a thread: the values are evaluated
// once per pair, and Dual<4> spills (1.8 to 2.7 KB a thread in the edge and
// shear terms). The whole call, its two solves included, takes 0.97 ms at
// 17 x 17 and 1.98 ms at 50 x 50 (2.57 and 3.39 when these kernels came, before
// the solves' present form); with forward-mode directions compressed by a
// 41-colouring over 128 copies of the cloths (512 directions of every element,
// 3.2 MB of workspace a node) it took 8.5 and 53.6 ms.
#include "ys_items.cuh"
#include "ys_kernels.cuh"

namespace ys {

namespace {

typedef Dual<2> D2;
constexpr int kEdgeVars = 15;   // dx 3, du, gx, a0 3, a1 3, e0, e1, rho, ks
constexpr int kEdgePairs = 8;
constexpr int kBendVars = 15;   // real: arms 6, du, kb; crimp: arms 6, kb
constexpr int kBendPairs = 8;   // 4 real, 4 crimp (the last input of those is unused)
constexpr int kFaceVars = 9;    // e1 3, e2 3, velocity sum 3
constexpr int kFacePairs = 5;
constexpr int kShearVars = 7;   // arms 6, SR
constexpr int kShearPairs = 4;
constexpr int kCrossVars = 8;   // comp, ce, mu, uvm, uvdot, FE, KEE, DEE
// fields a crossing keeps for the element kernels
constexpr int kC_FE = 0, kC_KEE = 2, kC_DEE = 4, kC_CL = 6, kC_CLE = 9, kC_N = 15, kC_UV = 18, kC_UVD = 20, kC_MU = 22;
static_assert(kC_MU + 1 == kAdjCrossFields, "crossing record");

// input i of a thread whose pair is `pair`
__device__ __forceinline__ D2 seed(double x, int i, int pair) {
  D2 d(x);
  d.d[0] = i == 2 * pair ? 1.0 : 0.0;
  d.d[1] = i == 2 * pair + 1 ? 1.0 : 0.0;
  return d;
}
// both derivatives of a pair, to fields `pair` of a record of nvar fields
__device__ __forceinline__ void keep(double* buf, int nvar, int pair, int64_t stride, int64_t at, const D2& phi) {
  for (int k = 0; k < 2; ++k)
    if (2 * pair + k < nvar) buf[(int64_t)(2 * pair + k) * stride + at] = phi.d[k];
}

// lambda and q at a node
struct Weights {
  const double* lam;
  const double* q;  // null: A carries no derivative
  int64_t nt;
  __device__ __forceinline__ double l(int c, int n) const { return lam[c * nt + n]; }
  __device__ __forceinline__ double x(int c, int n) const { return q ? q[c * nt + n] : 0.0; }
};

}  // namespace

// Cloth::update transposed. gin: [5 arrays] g' of LPos [3][nt], LVel [3][nt],
// EPos [2][nt], EVel [2][nt], EPosBar [2][nt] (component-major). Writes
// qbar [5][nt], the pass-through part of g (gout, same layout) and
// slide_bar [2][nt].
__global__ void k_adj_update(View v, AdjIO io, const double* q, double* qbar,
                             double* slide_bar) {
  chained();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= v.ntot) return;
  const int nt = v.ntot;
  const double h = v.h;
  const bool in = (v.flags[n] & YS_INTERIOR) != 0;
  for (int i = 0; i < 3; ++i) {
    const double gx = io.gin[0][i * nt + n], gv = io.gin[1][i * nt + n];
    qbar[i * nt + n] = gv + h * gx;  // V' = q, X' = X + h q
    io.gout[0][i * nt + n] = gx;
    io.gout[1][i * nt + n] = 0.0;
  }
  for (int k = 0; k < 2; ++k) {
    const double ge = io.gin[2][k * nt + n], gd = io.gin[3][k * nt + n], gb = io.gin[4][k * nt + n];
    io.gout[2][k * nt + n] = ge;
    io.gout[4][k * nt + n] = gb;
    if (in) {
      // EVel' = q_e, EPos' = EPos + h q_e, EPosBar' = EPosBar + slide q_e h
      const double s = v.SLIDE[k * nt + n], qe = q[(3 + k) * nt + n];
      qbar[(3 + k) * nt + n] = gd + h * ge + s * h * gb;
      io.gout[3][k * nt + n] = 0.0;
      slide_bar[k * nt + n] = gb * qe * h;
    } else {  // boundary crossings keep their Eulerian state
      qbar[(3 + k) * nt + n] = 0.0;
      io.gout[3][k * nt + n] = gd;
      slide_bar[k * nt + n] = 0.0;
    }
  }
}

// one thread per (pair, segment type, crossing)
__global__ void __launch_bounds__(64) k_adj_shear(View v, AdjWork w) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= (int64_t)kShearPairs * 4 * nt) return;
  const int ps = (int)(t / nt), n0 = (int)(t - (int64_t)ps * nt), pair = ps >> 2, seg = ps & 3;
  if (!(v.flags[n0] & YS_INTERIOR)) return;
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  const ShearIn<double> s = shear_load<double>(v, n0, seg);
  ShearIn<D2> d;
  for (int i = 0; i < 3; ++i) { d.d1[i] = seed(s.d1[i], i, pair); d.d3[i] = seed(s.d3[i], 3 + i, pair); }
  d.SR = seed(s.SR, 6, pair);
  d.jam = s.jam;
  const int n1 = n0 + shear_du(seg), n3 = n0 + shear_dv(seg) * P.W;
  const Weights W{w.lam, w.q, nt};
  double al[3], be[3], u[3], x[3];  // lambda and q of n1, n3 relative to n0
  for (int i = 0; i < 3; ++i) {
    al[i] = W.l(i, n1) - W.l(i, n0);
    be[i] = W.l(i, n3) - W.l(i, n0);
    u[i] = W.x(i, n1) - W.x(i, n0);
    x[i] = W.x(i, n3) - W.x(i, n0);
  }
  D2 phi = 0.0;
  shear_terms(d, P, v.h, v.trunc != 0, [&](int f, const D2& y) {
    double wt;
    if (f < kS_F3) wt = al[f];
    else if (f < kS_J11) wt = be[f - kS_F3];
    else {
      const int g = f - kS_J11, blk = g / 9, r = (g - 9 * blk) / 3, c = g - 9 * blk - 3 * r;  // J11, J13, J31, J33
      wt = -(blk < 2 ? al[r] : be[r]) * (blk == 0 || blk == 2 ? u[c] : x[c]);
    }
    phi += wt * y;
  });
  keep(w.shear, kShearVars, pair, 4LL * nt, (int64_t)seg * nt + n0, phi);
}

// Friction at a crossing: 32 crossings a block; four warps gather their sums
// (as k_cross), then each of two yarns' derivatives in two warps of two pairs
// each. comp and ce are the only inputs that lead to other elements.
__global__ void __launch_bounds__(128) k_adj_cross(View v, Records R, AdjWork w) {
  chained();
  __shared__ double sc[3][4][32], sk[6][4][32], sg[2][kCrossVars][32];
  const int m = threadIdx.x >> 5, i = threadIdx.x & 31;
  const int node = blockIdx.x * 32 + i;
  const bool valid = node < v.ntot;
  const int n = valid ? node : v.ntot - 1, nt = v.ntot;
  const NodeAt N(v, n);
  const bool on = valid && N.in;
  if (on) {
    CrossPart<double> c;
    cross_part(v, R, N, m, c);
    for (int r = 0; r < 3; ++r) { sc[r][m][i] = c.CL[r]; sk[r][m][i] = c.CLE[r]; }
    sk[3][m][i] = c.FE;
    sk[4][m][i] = c.KEE;
    sk[5][m][i] = c.DEE;
  }
  __syncthreads();
  double CL[3], cc = 0.0, nrm[3];
  const int k = m & 1, cl = v.node_cloth[n];
  const ClothParams& P = v.cp[cl];
  if (on) {
    double s[6], ce = 0.0;
    for (int r = 0; r < 3; ++r) {
      CL[r] = (sc[r][0][i] + sc[r][1][i]) + (sc[r][2][i] + sc[r][3][i]);
      nrm[r] = ld(v.NRM, r, nt, n);
      cc += nrm[r] * CL[r];
    }
    for (int r = 0; r < 6; ++r) s[r] = sk[r][2 * k][i] + sk[r][2 * k + 1][i];
    for (int r = 0; r < 3; ++r) ce += nrm[r] * s[r];
    const double comp = cc > 0.0 ? 0.5 * cc : 0.0;
    const double uvm = ld(v.UV, k, nt, n) - ld(v.UVB, k, nt, n), uvd = ld(v.UVD, k, nt, n);
    const double lam = w.lam[(3 + k) * (int64_t)nt + n], q = w.q ? w.q[(3 + k) * (int64_t)nt + n] : 0.0;
    const double sb = w.slide_bar[(int64_t)k * nt + n];
    for (int half = 0; half < 2; ++half) {
      const int pair = 2 * (m >> 1) + half;
      D2 slide, aEE, bE;
      friction_terms(P, v.h, v.trunc != 0, seed(comp, 0, pair), seed(0.5 * ce, 1, pair), seed(P.mu, 2, pair),
                     seed(uvm, 3, pair), seed(uvd, 4, pair), seed(s[3], 5, pair), seed(s[4], 6, pair),
                     seed(s[5], 7, pair), slide, aEE, bE);
      const D2 phi = lam * (bE - q * aEE) + sb * slide;
      sg[k][2 * pair][i] = phi.d[0];
      sg[k][2 * pair + 1][i] = phi.d[1];
    }
  }
  __syncthreads();
  if (m != 0 || !valid) return;
  auto put = [&](int f, double x) { w.cross[(int64_t)f * nt + n] = x; };
  if (!N.in) {
    for (int f = 0; f < kAdjCrossFields; ++f) put(f, 0.0);
    return;
  }
  // the compression also scales the crossing's shear segments
  double cb = sg[0][0][i] + sg[1][0][i];
  const double SR2 = P.S * (P.R * P.R);
  for (int seg = 0; seg < 4; ++seg) cb += SR2 * w.shear[(int64_t)6 * 4 * nt + (int64_t)seg * nt + n];
  const double hc = cc < 0.0 ? 0.0 : 0.5 * cb;  // comp = max(n . CL / 2, 0)
  for (int r = 0; r < 3; ++r) {
    double nb = hc * CL[r];
    put(kC_CL + r, hc * nrm[r]);
    for (int kk = 0; kk < 2; ++kk) {
      const double hk = 0.5 * sg[kk][1][i];
      put(kC_CLE + 3 * kk + r, hk * nrm[r]);
      nb += hk * (sk[r][2 * kk][i] + sk[r][2 * kk + 1][i]);
    }
    put(kC_N + r, nb);
  }
  for (int kk = 0; kk < 2; ++kk) {
    put(kC_FE + kk, sg[kk][5][i]);
    put(kC_KEE + kk, sg[kk][6][i]);
    put(kC_DEE + kk, sg[kk][7][i]);
    put(kC_UV + kk, sg[kk][3][i]);
    put(kC_UVD + kk, sg[kk][4][i]);
  }
  put(kC_MU, sg[0][2][i] + sg[1][2][i]);
}

// one thread per (pair, yarn direction, node): the edge starting at that node
__global__ void __launch_bounds__(64) k_adj_edge(View v, AdjWork w) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= (int64_t)kEdgePairs * 2 * nt) return;
  const int pk = (int)(t / nt), n0 = (int)(t - (int64_t)pk * nt), pair = pk >> 1, k = pk & 1;
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  if (k == 0 ? v.node_u[n0] >= P.W - 1 : v.node_v[n0] >= P.H - 1) return;
  const int n1 = n0 + (k == 0 ? 1 : P.W), nd[2] = {n0, n1};
  const EdgeIn<double> s = edge_load<double>(v, n0, n1, k);
  EdgeIn<D2> d;
  for (int i = 0; i < 3; ++i) {
    d.dx[i] = seed(s.dx[i], i, pair);
    d.a[0][i] = seed(s.a[0][i], 5 + i, pair);
    d.a[1][i] = seed(s.a[1][i], 8 + i, pair);
  }
  d.du = seed(s.du, 3, pair);
  d.gx = seed(s.gx, 4, pair);
  d.e[0] = seed(s.e[0], 11, pair);
  d.e[1] = seed(s.e[1], 12, pair);
  d.rho = seed(s.rho, 13, pair);
  d.ks = seed(s.ks, 14, pair);
  d.in[0] = s.in[0];
  d.in[1] = s.in[1];
  d.over = s.over;
  const Weights W{w.lam, w.q, nt};
  double l[2][4], q[2][4];
  for (int a = 0; a < 2; ++a)
    for (int i = 0; i < 4; ++i) {
      l[a][i] = W.l(i < 3 ? i : 3 + k, nd[a]);
      q[a][i] = W.x(i < 3 ? i : 3 + k, nd[a]);
    }
  auto cr = [&](int f, int a) { return w.cross[(int64_t)f * nt + nd[a]]; };
  D2 phi = 0.0, lP, cl, cle, lx = 0.0, xx = 0.0;
  double al[3], u[3];
  for (int i = 0; i < 3; ++i) { al[i] = l[1][i] - l[0][i]; u[i] = q[1][i] - q[0][i]; }
  edge_terms(d, P, k, v.h, v.trunc != 0, [&](int f, const D2& y) {
    if (f == kE_cl) cl = y;
    else if (f == kE_cle) cle = y;
    else if (f == kE_lP) {
      lP = y;
      phi -= (al[0] * u[0] + al[1] * u[1] + al[2] * u[2]) * y;  // lP (I - d d^T) between the ends' differences
    } else if (f >= kE_d && f < kE_le) {
      const int i = f - kE_d;
      lx += al[i] * y;
      xx += u[i] * y;
      phi += (cl * (cr(kC_CL + i, 0) - cr(kC_CL + i, 1))) * y;
      phi += (cle * ((s.in[0] ? cr(kC_CLE + 3 * k + i, 0) : 0.0) + (s.in[1] ? cr(kC_CLE + 3 * k + i, 1) : 0.0))) * y;
      if (i == 2) phi += lP * (lx * xx);
    } else {
      double wt;
      if (f < kE_lP) {  // iso blocks
        const int a = f >> 1, c = f & 1;
        wt = -(l[a][0] * q[c][0] + l[a][1] * q[c][1] + l[a][2] * q[c][2]);
      } else if (f < kE_el) {
        const int p = (f - kE_le) / 3, i = f - kE_le - 3 * p;
        wt = -l[p >> 1][i] * q[p & 1][3];
      } else if (f < kE_ee) {
        const int p = (f - kE_el) / 3, i = f - kE_el - 3 * p;
        wt = -l[p >> 1][3] * q[p & 1][i];
      } else if (f < kE_b) {
        const int p = f - kE_ee;
        wt = -l[p >> 1][3] * q[p & 1][3];
      } else if (f < kE_fe) {
        wt = l[(f - kE_b) >> 2][(f - kE_b) & 3];
      } else if (f < kE_kee) {
        wt = cr(kC_FE + k, f - kE_fe);
      } else if (f < kE_dee) {
        wt = cr(kC_KEE + k, f - kE_kee);
      } else {
        wt = cr(kC_DEE + k, f - kE_dee);
      }
      phi += wt * y;
    }
  });
  keep(w.edge, kEdgeVars, pair, 2LL * nt, (int64_t)k * nt + n0, phi);
}

// one thread per (pair, yarn direction, middle node)
__global__ void __launch_bounds__(64) k_adj_bend(View v, AdjWork w) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= (int64_t)kBendPairs * 2 * nt) return;
  const int pk = (int)(t / nt), n0 = (int)(t - (int64_t)pk * nt), pair = pk >> 1, k = pk & 1;
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  const int pos = k == 0 ? v.node_u[n0] : v.node_v[n0], len = k == 0 ? P.W : P.H;
  if (pos < 1 || pos > len - 2) return;
  const int step = k == 0 ? 1 : P.W, n1 = n0 + step, n2 = n0 - step;
  const int line = k == 0 ? P.warp_line_off + v.node_v[n0] : P.weft_line_off + v.node_u[n0];
  const double kb = v.line_kb[line];
  const bool in0 = (v.flags[n0] & YS_INTERIOR) != 0, in1 = (v.flags[n1] & YS_INTERIOR) != 0,
             in2 = (v.flags[n2] & YS_INTERIOR) != 0;
  auto cr = [&](int f, int n) { return w.cross[(int64_t)f * nt + n]; };
  D2 phi = 0.0;
  if (pair < 4) {
    D2 to1[3], to2[3];
    for (int i = 0; i < 3; ++i) {
      const double x0 = ld(v.X, i, nt, n0);
      to1[i] = seed(ld(v.X, i, nt, n1) - x0, i, pair);
      to2[i] = seed(ld(v.X, i, nt, n2) - x0, 3 + i, pair);
    }
    const D2 du = seed(ld(v.UV, k, nt, n1) - ld(v.UV, k, nt, n2), 6, pair), kbd = seed(kb, 7, pair);
    const Weights W{w.lam, w.q, nt};
    const double h = v.h, mh2 = -(v.h * v.h);
    const int e = 3 + k;
    const double le0 = W.l(e, n0), le1 = W.l(e, n1), le2 = W.l(e, n2);
    const double qe1 = W.x(e, n1), qe2 = W.x(e, n2);
    double al[3], be[3], u[3], x[3], m1[3], m2[3];
    for (int i = 0; i < 3; ++i) {
      const double l0 = W.l(i, n0), l1 = W.l(i, n1), l2 = W.l(i, n2), q0 = W.x(i, n0), q1 = W.x(i, n1), q2 = W.x(i, n2);
      al[i] = l1 - l0;
      be[i] = l2 - l0;
      u[i] = q1 - q0;
      x[i] = q2 - q0;
      // weights of -h^2 F1 / du, -h^2 F2 / du in the Eulerian couplings (row_part)
      double both = 0.0;
      if (in0 && in2) both += l0 * qe2 + le0 * q2;
      if (in0 && in1) both -= l0 * qe1 + le1 * q0;
      m2[i] = (in2 ? l2 * qe2 + le2 * q2 : 0.0) - both;
      m1[i] = -(in1 ? l1 * qe1 + le1 * q1 : 0.0) - both;
    }
    const double wE = -mh2 * ((in2 ? le2 * qe2 : 0.0) + (in1 ? le1 * qe1 : 0.0)) + (in2 ? cr(kC_KEE + k, n2) : 0.0) +
                      (in1 ? cr(kC_KEE + k, n1) : 0.0);
    const double wF = (in2 ? h * le2 + cr(kC_FE + k, n2) : 0.0) - (in1 ? h * le1 + cr(kC_FE + k, n1) : 0.0);
    D2 idu;
    bend_real(to1, to2, du, kbd, h, [&](int f, const D2& y) {
      if (f == kB_idu) idu = y;
      else if (f == kB_E1E1) phi += wE * y;
      else if (f == kB_Fu2) phi += wF * y;
      else if (f >= kB_F1 && f < kB_F2) phi += (h * al[f - kB_F1] - (mh2 * m1[f - kB_F1]) * idu) * y;
      else if (f >= kB_F2 && f < kB_idu) phi += (h * be[f - kB_F2] - (mh2 * m2[f - kB_F2]) * idu) * y;
      else if (f < kB_L12) {
        const bool one = f < kB_L22;
        const int g = one ? f : f - kB_L22;
        const int i = g < 3 ? 0 : g < 5 ? 1 : 2, j = g < 3 ? g : g < 5 ? g - 2 : 2;
        const double *a = one ? al : be, *b = one ? u : x;
        phi -= (i == j ? a[i] * b[i] : a[i] * b[j] + a[j] * b[i]) * y;
      } else {
        const int i = (f - kB_L12) / 3, j = f - kB_L12 - 3 * i;
        phi -= (be[i] * u[j] + al[j] * x[i]) * y;
      }
    });
    keep(w.bend, 8, pair, 2LL * nt, (int64_t)k * nt + n0, phi);
  } else {
    const int cp = pair - 4;
    double c0[3], c1[3], c2[3];
    crimp_point(v, n0, k, c0);
    crimp_point(v, n1, k, c1);
    crimp_point(v, n2, k, c2);
    D2 to1[3], to2[3];
    for (int i = 0; i < 3; ++i) { to1[i] = seed(c1[i] - c0[i], i, cp); to2[i] = seed(c2[i] - c0[i], 3 + i, cp); }
    const double icu = crimp_icu(v, n2, n1, k), sgn = k == 0 ? 1.0 : -1.0;
    bend_crimp(to1, to2, icu, seed(kb, 6, cp), [&](int f, const D2& y) {
      if (f == kB_cidu) return;
      const bool one = f < kB_cF2;
      const int i = f - (one ? kB_cF1 : kB_cF2), n = one ? n1 : n2;
      const double ce = icu * cr(kC_CLE + 3 * k + i, n);
      phi += (sgn * (cr(kC_CL + i, n) - cr(kC_CL + i, n0) + (one ? -ce : ce))) * y;
    });
    keep(w.bend + 8LL * 2 * nt, 7, cp, 2LL * nt, (int64_t)k * nt + n0, phi);
  }
}

// one thread per (pair, face of a cell, cell)
__global__ void __launch_bounds__(64) k_adj_face(View v, AdjWork w) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= (int64_t)kFacePairs * 2 * nt) return;
  const int pf = (int)(t / nt), tl = (int)(t - (int64_t)pf * nt), pair = pf >> 1, which = pf & 1;
  const ClothParams& P = v.cp[v.node_cloth[tl]];
  if (v.node_u[tl] >= P.W - 1 || v.node_v[tl] >= P.H - 1) return;
  int n[3];
  cell_face(v, tl, which, n);
  D2 e1[3], e2[3], vs[3], f3[3], phi = 0.0;
  for (int i = 0; i < 3; ++i) {
    const double xa = ld(v.X, i, nt, n[0]);
    e1[i] = seed(ld(v.X, i, nt, n[1]) - xa, i, pair);
    e2[i] = seed(ld(v.X, i, nt, n[2]) - xa, 3 + i, pair);
    vs[i] = seed(ld(v.V, i, nt, n[0]) + ld(v.V, i, nt, n[1]) + ld(v.V, i, nt, n[2]), 6 + i, pair);
  }
  wind_terms(P, e1, e2, vs, f3);
  for (int i = 0; i < 3; ++i) {
    const double l = w.lam[(int64_t)i * nt + n[0]] + w.lam[(int64_t)i * nt + n[1]] + w.lam[(int64_t)i * nt + n[2]];
    phi += (v.h * l) * f3[i];
  }
  keep(w.face, kFaceVars, pair, 2LL * nt, (int64_t)which * nt + tl, phi);
}

// The normal's adjoint at an interior crossing (friction's, and the crimp
// offsets' of the up to six bend segments it is part of) carried to the
// scatter matrix: with eigenpairs (l_j, v_j) and the normal n = +-v_m, phi changes
// by g^T dS n, g = sum_{j != m} (n_bar . v_j) / (l_m - l_j) v_j
// (node_normal_dual's perturbation, transposed). Writes g, n and the crossing's
// mean; k_adj_gather forms the five positions' shares.
__global__ void __launch_bounds__(128) k_adj_normal(View v, const int* __restrict__ nodes, int count, AdjWork w) {
  chained();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int n = nodes[t], nt = v.ntot;
  const NodeAt N(v, n);
  const double R = v.cp[v.node_cloth[n]].R;
  double nb[3];
  for (int r = 0; r < 3; ++r) nb[r] = w.cross[(int64_t)(kC_N + r) * nt + n];
  const double* cb = w.bend + 8LL * 2 * nt;  // crimp arms
  for (int k = 0; k < 2; ++k) {
    const double sg = k == 0 ? -R : R;
    const int step = N.step(k), pos = N.pos(k), len = N.len(k);
    auto g = [&](int f, int mid) { return cb[(int64_t)f * 2 * nt + (int64_t)k * nt + mid]; };
    for (int r = 0; r < 3; ++r) {
      double s = 0.0;
      s -= g(r, n) + g(3 + r, n);                          // middle (an interior crossing is one)
      if (pos + 1 <= len - 2) s += g(3 + r, n + step);     // n2 of the next segment
      if (pos - 1 >= 1) s += g(r, n - step);               // n1 of the last
      nb[r] += sg * s;
    }
  }
  const int ids[5] = {n, n - 1, n + 1, n - N.W, n + N.W};
  double p[5][3], mean[3] = {0, 0, 0}, S[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, nn[3], g[3];
  for (int m = 0; m < 5; ++m)
    for (int i = 0; i < 3; ++i) { p[m][i] = ld(v.X, i, nt, ids[m]); mean[i] += p[m][i]; }
  for (int i = 0; i < 3; ++i) mean[i] /= 5.0;
  for (int m = 0; m < 5; ++m)
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) S[i][j] += (p[m][i] - mean[i]) * (p[m][j] - mean[j]);
  for (int i = 0; i < 3; ++i) nn[i] = ld(v.NRM, i, nt, n);
  NormalResponse(S, nn).respond(nb, g);
  for (int i = 0; i < 3; ++i) {
    w.normal[(int64_t)i * nt + n] = g[i];
    w.normal[(int64_t)(3 + i) * nt + n] = nn[i];
    w.normal[(int64_t)(6 + i) * nt + n] = mean[i];
  }
}

// adds every element's share to node n's state adjoints, in a fixed order;
// one thread per (component, node): x, y, z and the two yarns
__global__ void __launch_bounds__(128) k_adj_gather(View v, AdjWork w, AdjIO io) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= 5LL * nt) return;
  const int comp = (int)(t / nt), n = (int)(t - (int64_t)comp * nt);
  const NodeAt N(v, n);
  const ClothParams& P = v.cp[v.node_cloth[n]];
  auto E = [&](int f, int k, int a) { return w.edge[(int64_t)f * 2 * nt + (int64_t)k * nt + a]; };
  auto Bn = [&](int f, int k, int a) { return w.bend[(int64_t)f * 2 * nt + (int64_t)k * nt + a]; };
  if (comp >= 3) {  // EPos, EVel, EPosBar along yarn k
    const int k = comp - 3, step = N.step(k), pos = N.pos(k), len = N.len(k);
    double gu = w.cross[(int64_t)(kC_UV + k) * nt + n], gd = w.cross[(int64_t)(kC_UVD + k) * nt + n];
    io.gout[4][(int64_t)k * nt + n] -= gu;
    if (pos < len - 1) { gu -= E(3, k, n); gd += E(11, k, n); }
    if (pos > 0) { gu += E(3, k, n - step); gd += E(12, k, n - step); }
    if (pos + 1 <= len - 2) gu -= Bn(6, k, n + step);  // n2 of the next segment
    if (pos - 1 >= 1) gu += Bn(6, k, n - step);        // n1 of the last
    io.gout[2][(int64_t)k * nt + n] += gu;
    io.gout[3][(int64_t)k * nt + n] += gd;
    return;
  }
  const int r = comp;
  double gx = 0.0, gv = 0.0;
  for (int k = 0; k < 2; ++k) {
    const int step = N.step(k), pos = N.pos(k), len = N.len(k);
    if (pos < len - 1) { gx += P.G[r] * E(4, k, n) - E(r, k, n); gv += E(5 + r, k, n); }
    if (pos > 0) { gx += P.G[r] * E(4, k, n - step) + E(r, k, n - step); gv += E(8 + r, k, n - step); }
    for (int part = 0; part < 2; ++part) {  // real arms, crimp arms
      const int f = 8 * part + r;
      if (pos >= 1 && pos <= len - 2) gx -= Bn(f, k, n) + Bn(f + 3, k, n);
      if (pos + 1 >= 1 && pos + 1 <= len - 2) gx += Bn(f + 3, k, n + step);
      if (pos - 1 >= 1 && pos - 1 <= len - 2) gx += Bn(f, k, n - step);
    }
  }
  for (int m = 0; m < 4; ++m) {  // faces of the cells around the node
    const int ci = N.u - 1 + (m & 1), cj = N.w - 1 + (m >> 1);
    if (ci < 0 || ci >= N.W - 1 || cj < 0 || cj >= N.H - 1) continue;
    const int tl = n + (ci - N.u) + (cj - N.w) * N.W;
    for (int which = 0; which < 2; ++which) {
      int fn[3];
      cell_face(v, tl, which, fn);
      auto F = [&](int f) { return w.face[(int64_t)f * 2 * nt + (int64_t)which * nt + tl]; };
      if (n == fn[0]) gx -= F(r) + F(3 + r);
      else if (n == fn[1]) gx += F(r);
      else if (n == fn[2]) gx += F(3 + r);
      else continue;
      gv += F(6 + r);
    }
  }
  for (int seg = 0; seg < 4; ++seg) {
    const int du = shear_du(seg), dv = shear_dv(seg);
    auto S = [&](int f, int a) { return w.shear[(int64_t)f * 4 * nt + (int64_t)seg * nt + a]; };
    if (N.in) gx -= S(r, n) + S(3 + r, n);
    if (N.interior(N.u - du, N.w)) gx += S(r, n - du);
    if (N.interior(N.u, N.w - dv)) gx += S(3 + r, n - dv * N.W);
  }
  // normals of the node and its yarn neighbours: g (r . n) + n (g . r)
  const double x[3] = {ld(v.X, 0, nt, n), ld(v.X, 1, nt, n), ld(v.X, 2, nt, n)};
  for (int m = 0; m < 5; ++m) {
    const int du = m == 1 ? -1 : m == 2 ? 1 : 0, dv = m == 3 ? -1 : m == 4 ? 1 : 0;
    if (!N.interior(N.u + du, N.w + dv)) continue;
    const int j = n + du + dv * N.W;
    double rn = 0.0, rg = 0.0;
    for (int i = 0; i < 3; ++i) {
      const double rr = x[i] - w.normal[(int64_t)(6 + i) * nt + j];
      rg += rr * w.normal[(int64_t)i * nt + j];
      rn += rr * w.normal[(int64_t)(3 + i) * nt + j];
    }
    gx += w.normal[(int64_t)r * nt + j] * rn + w.normal[(int64_t)(3 + r) * nt + j] * rg;
  }
  if (v.flags[n] & YS_FIXED) gx -= v.h * P.kh * w.lam[(int64_t)r * nt + n];
  io.gout[0][(int64_t)r * nt + n] += gx;
  io.gout[1][(int64_t)r * nt + n] += gv;
}

constexpr int kParamThreads = 256;
// material adjoints: rho, Y, B of every line, one warp each, over the line's
// edges and bend segments (ks, kb = (Y, B) a, a = pi R^2), S and mu of every
// cloth, one block each (one warp took 97 us over a 50 x 50 cloth's crossings)
__global__ void __launch_bounds__(kParamThreads) k_adj_params(View v, AdjWork w, const double* __restrict__ line_a,
                                                    const int* __restrict__ line_cloth, AdjParamOut gp) {
  chained();
  __shared__ double sh[2][kParamThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nl = v.nlines, nt = v.ntot;
  if ((int)blockIdx.x >= v.ncloth) {
    const int id = (blockIdx.x - v.ncloth) * (kParamThreads / 32) + wid;
    if (id >= nl) return;
    const ClothParams& P = v.cp[line_cloth[id]];
    const bool weft = id >= P.weft_line_off;
    const int k = weft ? 1 : 0, at = weft ? id - P.weft_line_off : id - P.warp_line_off;
    const int first = P.node_off + (weft ? at : at * P.W), step = weft ? P.W : 1, len = weft ? P.H : P.W;
    double s[3] = {0.0, 0.0, 0.0};
    for (int i = lane; i < len; i += 32) {
      const int64_t o = (int64_t)k * nt + first + i * step, st2 = 2LL * nt;
      if (i < len - 1) { s[0] += w.edge[13 * st2 + o]; s[1] += w.edge[14 * st2 + o]; }
      if (i >= 1 && i <= len - 2) s[2] += w.bend[7 * st2 + o] + w.bend[14 * st2 + o];
    }
    for (int p = 0; p < 3; ++p) {
      const double x = cloth_tree(s[p]);
      if (lane == 0) gp.line[p][id] = p == 0 ? x : x * line_a[id];
    }
  } else {
    const int c = blockIdx.x;
    const ClothParams& P = v.cp[c];
    double sS = 0.0, sm = 0.0;
    for (int i = threadIdx.x; i < P.W * P.H; i += kParamThreads) {
      const int n = P.node_off + i;
      sm += w.cross[(int64_t)kC_MU * nt + n];
      if (!(v.flags[n] & YS_INTERIOR)) continue;
      double a = 0.0;
      for (int seg = 0; seg < 4; ++seg) a += w.shear[(int64_t)6 * 4 * nt + (int64_t)seg * nt + n];
      sS += (v.COMP[n] + 1.0) * (P.R * P.R) * a;
    }
    sS = cloth_tree(sS);
    sm = cloth_tree(sm);
    if (lane == 0) { sh[0][wid] = sS; sh[1][wid] = sm; }
    __syncthreads();
    if (threadIdx.x < 2) {
      double x = 0.0;
      for (int i = 0; i < kParamThreads / 32; ++i) x += sh[threadIdx.x][i];
      gp.cloth[threadIdx.x][c] = x;
    }
  }
}

// dL/d ext = h lambda on the components the gather adds ext to (x, y, z of
// every node, u, v of interior crossings); node layout [nt][5]
__global__ void k_adj_ext(View v, const double* lambda, double* gext) {
  chained();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= v.ntot) return;
  const bool in = (v.flags[n] & YS_INTERIOR) != 0;
  for (int c = 0; c < 5; ++c) gext[(int64_t)n * 5 + c] = (c < 3 || in) ? v.h * lambda[(int64_t)c * v.ntot + n] : 0.0;
}

static inline unsigned nbl(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

AdjSizes adjoint_sizes() {
  return AdjSizes{(int64_t)kEdgeVars * 2, (int64_t)kBendVars * 2, (int64_t)kFaceVars * 2, (int64_t)kShearVars * 4,
                  kAdjCrossFields, 9};
}

void launch_adj_update(const View& v, const AdjIO& io, const double* q, double* qbar, double* slide_bar,
                       cudaStream_t s) {
  chain(k_adj_update, nbl(v.ntot, 256), 256, s, v, io, q, qbar, slide_bar);
}
int launch_adj_vjp(const View& v, const Records& R, const AdjWork& w, const int* interior, int n_interior,
                   const AdjIO& io, const double* line_a, const int* line_cloth, const AdjParamOut& gp,
                   cudaStream_t s) {
  const int64_t nt = v.ntot;
  chain(k_adj_shear, nbl(kShearPairs * 4 * nt, 64), 64, s, v, w);
  chain(k_adj_cross, nbl(nt, 32), 128, s, v, R, w);
  chain(k_adj_edge, nbl(kEdgePairs * 2 * nt, 64), 64, s, v, w);
  chain(k_adj_bend, nbl(kBendPairs * 2 * nt, 64), 64, s, v, w);
  chain(k_adj_face, nbl(kFacePairs * 2 * nt, 64), 64, s, v, w);
  chain(k_adj_normal, nbl(n_interior, 128), 128, s, v, interior, n_interior, w);
  chain(k_adj_gather, nbl(5 * nt, 128), 128, s, v, w, io);
  chain(k_adj_params, v.ncloth + nbl(v.nlines, kParamThreads / 32), kParamThreads, s, v, w, line_a, line_cloth, gp);
  return 8;
}
void launch_adj_ext(const View& v, const double* lambda, double* gext, cudaStream_t s) {
  chain(k_adj_ext, nbl(v.ntot, 256), 256, s, v, lambda, gext);
}

}  // namespace ys
