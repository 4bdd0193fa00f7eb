// ys_physics.cuh -- per-element yarn forces and Jacobians of one implicit step.
//
// Each routine handles one element (edge, bend segment, crossing, shear
// segment, face) and returns its contribution to the step's system
//     A = M - h^2 dF/dx - h dF/dv,   b = h (F - (dF/dv)^T v) + M v
// (src/TrainHelper.cpp:19-20). The record producers (ys_kernels.cu)
// write each element's contribution to its own record, and the per-node
// gathers (ys_items.cuh) sum a node's records in a fixed order into the
// structured stencil layout of ys_common.cuh, so the accumulation is
// deterministic without atomics.
//
// The arithmetic restates the reference's hand-derived expressions term by
// term, including the places where they differ from exact derivatives; every
// routine names the reference lines it follows. The edge kinetic-energy terms
// are evaluated in closed form: with qdot = (a0, e0, a1, e1) and the 8x8 edge
// mass matrix built from 4x4 blocks B = [[z I, p], [q^T, s]] as
// [[2B, B], [B, 2B]], every quadratic form reduces to
//     qdot^T [[2B,B],[B,2B]] qdot = z Saa + p.Sae + q.Sea + s See
// and every product [[2B,B],[B,2B]] qdot = (B m0, B m1) with m0 = 2v0 + v1,
// m1 = v0 + 2v1, so no 8x8 matrix is ever formed.
#pragma once

#include <math.h>

#include "ys_common.cuh"
#include "ys_dual.cuh"

namespace ys {

// ---------------------------------------------------------------- helpers
template <class T>
YS_HD T dot3(const T* a, const T* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
template <class T>
YS_HD T norm3(const T* a) { return sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]); }
template <class T>
YS_HD void cross3(const T* a, const T* b, T* o) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}
// 1 / sqrt(x): one device instruction sequence instead of a square root and a
// division (1 ulp)
YS_HD double rsqrt_(double x) {
#if defined(__CUDA_ARCH__)
  return ::rsqrt(x);
#else
  return 1.0 / ::sqrt(x);
#endif
}
template <int K>
YS_HD Dual<K> rsqrt_(const Dual<K>& a) {
  const double r = rsqrt_(a.v);
  return chain(a, r, -0.5 * r * (r * r));
}
// x / l from l and il = 1 / l, correctly rounded but for rare ties: the
// product and its residual, two operations more than the bare product. An
// axis-aligned x gives exactly +-1 (x = l), as a division does.
YS_HD double quot(double x, double l, double il) {
  const double q = x * il;
  return fma(fma(-q, l, x), il, q);
}
template <int K>
YS_HD Dual<K> quot(const Dual<K>& x, const Dual<K>& l, const Dual<K>& il) {
  Dual<K> r;
  r.v = quot(x.v, l.v, il.v);
  for (int k = 0; k < K; ++k) r.d[k] = (x.d[k] - r.v * l.d[k]) * il.v;
  return r;
}
// sqrt(x) from x and ix = 1 / sqrt(x), correctly rounded but for rare ties
YS_HD double root(double x, double ix) {
  const double l = x * ix;
  return fma(fma(-l, l, x), 0.5 * ix, l);
}
template <int K>
YS_HD Dual<K> root(const Dual<K>& x, const Dual<K>& ix) {
  return chain(x, root(x.v, ix.v), 0.5 * ix.v);
}
YS_HD double ld(const double* p, int comp, int ntot, int node) { return p[(int64_t)comp * ntot + node]; }
YS_HD double& st(double* p, int comp, int ntot, int node) { return p[(int64_t)comp * ntot + node]; }

// Scalar-generic loads and stores. A per-node array p holds comp c of node i
// at p[c * ntot + i]; its tangent array dp (forward-mode runs only) holds
// tangent k at dp[(c * kTangents + k) * ntot + i]; a Dual of fewer directions
// reads those from dp on. Record buffers use the same rule with c = field *
// nslot + slot. With T = double the tangent arrays are never touched.
YS_HD void lds(const double* p, const double* dp, int c, int ntot, int i, double& x) {
  (void)dp;
  x = p[(int64_t)c * ntot + i];
}
template <int K>
YS_HD void lds(const double* p, const double* dp, int c, int ntot, int i, Dual<K>& x) {
  x.v = p[(int64_t)c * ntot + i];
  for (int k = 0; k < K; ++k) x.d[k] = dp ? dp[((int64_t)c * kTangents + k) * ntot + i] : 0.0;
}
template <class T>
YS_HD T ldT(const double* p, const double* dp, int c, int ntot, int i) {
  T x;
  lds(p, dp, c, ntot, i, x);
  return x;
}
YS_HD void stT(double* p, double* dp, int c, int ntot, int i, const double& x) {
  (void)dp;
  p[(int64_t)c * ntot + i] = x;
}
template <int K>
YS_HD void stT(double* p, double* dp, int c, int ntot, int i, const Dual<K>& x) {
  p[(int64_t)c * ntot + i] = x.v;
  if (dp)
    for (int k = 0; k < K; ++k) dp[((int64_t)c * kTangents + k) * ntot + i] = x.d[k];
}
// a parameter of index i in a table of n entries (tangent k at dp[k * n + i])
YS_HD void ldp(const double* p, const double* dp, int i, int n, double& x) {
  (void)dp;
  (void)n;
  x = p[i];
}
template <int K>
YS_HD void ldp(const double* p, const double* dp, int i, int n, Dual<K>& x) {
  x.v = p[i];
  for (int k = 0; k < K; ++k) x.d[k] = dp ? dp[(int64_t)k * n + i] : 0.0;
}
template <class T>
YS_HD T ldpT(const double* p, const double* dp, int i, int n) {
  T x;
  ldp(p, dp, i, n, x);
  return x;
}
// per-cloth parameters S and mu (values in ClothParams, tangents [K][ncloth])
template <class T>
YS_HD T cloth_S(const View& v, int c) { return ldpT<T>(&v.cp[c].S, v.dS ? v.dS + c : nullptr, 0, v.ncloth); }
template <class T>
YS_HD T cloth_mu(const View& v, int c) { return ldpT<T>(&v.cp[c].mu, v.dmu ? v.dmu + c : nullptr, 0, v.ncloth); }

// ------------------------------------------------------------ edge element
// Local DOFs of an edge: x0 (0..2), e0 (3), x1 (4..6), e1 (7), where e is the
// Eulerian coordinate along the edge's yarn (u for warp, v for weft); blocks
// are indexed p = 2 * (row node) + (column node). Every node-node block is
// iso I + s lP (I - d d^T) with s = +1 on the diagonal and -1 across (mass,
// inertia and dM/dt blocks are multiples of I, stretch adds the projector).
//
// The record of an edge: what the gathers read of it.
constexpr int kE_llI = 0;   // [4]     iso of A[x(n_a)][x(n_b)]
constexpr int kE_lP = 4;    //         -h^2 ks / l
constexpr int kE_d = 5;     // [3]     edge direction
constexpr int kE_le = 8;    // [4][3]  A[x(n_a)][e(n_b)]
constexpr int kE_el = 20;   // [4][3]  A[e(n_a)][x(n_b)]
constexpr int kE_ee = 32;   // [4]     A[e(n_a)][e(n_b)]
constexpr int kE_b = 36;    // [8]     contribution to b
constexpr int kE_fe = 44;   // [2]     F_E before friction
constexpr int kE_kee = 46;  // [2]     dF_E/dE, position
constexpr int kE_dee = 48;  // [2]     dF_E/dE, velocity
constexpr int kE_cl = 50;   //         crimp compression: +cl d at n0, -cl d at n1
constexpr int kE_cle = 51;  //         its Eulerian derivative: cle d at the interior ends, of the sign of du
constexpr int kEdgeFields = 52;

template <class T>
struct EdgeOut {
  T f[kEdgeFields];
};

// All terms of one edge (src/PhysicsCloth.cpp:64-80): Mass (250-338), Gravity
// (340-425), Stretch (427-577), ParaColli (989-1069), Inertia (1071-1901) and
// MDotVDot (1903-2577), forces and both Jacobians, as they enter
// A = M - h^2 K - h D and b = h F + (M - h D^T) V; put(field, value) receives
// each field of the record once.
//
// With w = dx / du, m0 = 2 a0 + a1, m1 = a0 + 2 a1 (mu0, mu1 the same of the
// Eulerian velocities), S = a0 mu0 + a1 mu1, D = a1 - a0 and delta = e1 - e0,
// the reference's expressions collapse: both mixed sums of its quadratic form
// equal S; Inertia's forces are r6 (S - See w) and r6 (w.w See - a.Ma) / 2;
// B_M m and B_dot m of MDotVDot combine to r_b = r6 (delta m_b - mu_b D); the
// node-node part of MDotVDot_D_Pos cancels; the two velocity Jacobians add to
// multiples of m, D and mu w. Every block is then a few multiples of S, w, D,
// m and G. Its quirks are kept: the sign-asymmetric mixed block of
// Inertia_D_Pos (1357-1361; the +1 / -3 below), MDotVDot_D_Pos added and with
// the squared r6 of "- rho / 6 r" (2154-2234), ParaColli_D proportional to the
// overlap itself. Term by term as the reference writes them, an edge took
// 1,690 FP64 operations; this form takes about 500 (on 255,292 nodes 453 us for
// 1,044; 443 with |w| rounded once less, see nw).
// One edge's inputs: dx = x1 - x0, gx = G . (x0 + x1), the velocities a and e
// of its ends, du, and the yarn's density and stretch stiffness.
template <class T>
struct EdgeIn {
  T dx[3], gx, a[2][3], du, e[2], rho, ks;
  bool in[2];  // interior ends
  bool over;   // the yarn changes side between them
};
template <class T>
YS_HD EdgeIn<T> edge_load(const View& v, int n0, int n1, int k) {
  const int nt = v.ntot;
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  EdgeIn<T> s;
  const uint8_t f0 = v.flags[n0], f1 = v.flags[n1];
  s.in[0] = (f0 & YS_INTERIOR) != 0;
  s.in[1] = (f1 & YS_INTERIOR) != 0;
  s.over = ((f0 & YS_FLIP) != 0) != ((f1 & YS_FLIP) != 0);
  const int line = (k == 0) ? P.warp_line_off + v.node_v[n0] : P.weft_line_off + v.node_u[n0];
  s.rho = ldpT<T>(v.line_rho, v.dline_rho, line, v.nlines);
  s.ks = ldpT<T>(v.line_ks, v.dline_ks, line, v.nlines);
  s.gx = 0.0;
  for (int i = 0; i < 3; ++i) {
    const T x0 = ldT<T>(v.X, v.dX, i, nt, n0), x1 = ldT<T>(v.X, v.dX, i, nt, n1);
    s.dx[i] = x1 - x0;
    s.gx += P.G[i] * (x0 + x1);
    s.a[0][i] = ldT<T>(v.V, v.dV, i, nt, n0);
    s.a[1][i] = ldT<T>(v.V, v.dV, i, nt, n1);
  }
  s.du = ldT<T>(v.UV, v.dUV, k, nt, n1) - ldT<T>(v.UV, v.dUV, k, nt, n0);
  s.e[0] = ldT<T>(v.UVD, v.dUVD, k, nt, n0);
  s.e[1] = ldT<T>(v.UVD, v.dUVD, k, nt, n1);
  return s;
}
template <class T, class Put>
YS_HD void edge_terms(const EdgeIn<T>& s, const ClothParams& P, int k, double h, bool trunc, Put&& put) {
  const bool* in = s.in;
  const bool both = in[0] && in[1];
  const T &rho = s.rho, &ks = s.ks, &du = s.du, &gx = s.gx;
  const T(&dx)[3] = s.dx;
  const T(&a)[2][3] = s.a;
  const T(&e)[2] = s.e;
  const double mh2 = -(h * h);
  const T idu = 1.0 / du, aidu = fabs(idu);
  const T d2 = dot3(dx, dx), il = rsqrt_(d2);
  T w[3], d[3];
  for (int i = 0; i < 3; ++i) { w[i] = dx[i] * idu; d[i] = dx[i] * il; }
  // |w|, rounded as a square root and a division: exactly 1 at rest, whatever
  // the spacing, so that a resting yarn has no stretch force
  const T nw = quot(root(d2, il), T(fabs(du)), aidu);
  const T ww = nw * nw;
  const T r6 = (1.0 / 6.0) * rho, q = r6 * du;
  const T zero = T(0.0);
  // ---- stretch scalars; the crimp accumulators
  const T strf = ks * (nw - 1.0), ksw = ks * aidu, ksi = ks * idu;
  {
    const double sgn = (k == 0) ? 1.0 : -1.0;
    put(kE_cl, sgn * strf);
    put(kE_cle, sgn * (ksi * nw));
    put(kE_lP, mh2 * (ks * il));
    for (int i = 0; i < 3; ++i) put(kE_d + i, d[i]);
  }
  // ---- shared kinetic sums
  T m[2][3], mu[2], D[3];
  for (int i = 0; i < 3; ++i) {
    m[0][i] = 2.0 * a[0][i] + a[1][i];
    m[1][i] = a[0][i] + 2.0 * a[1][i];
    D[i] = a[1][i] - a[0][i];
  }
  mu[0] = 2.0 * e[0] + e[1];
  mu[1] = e[0] + 2.0 * e[1];
  const T dl = e[1] - e[0], See = e[0] * mu[0] + e[1] * mu[1];
  const T wD = dot3(w, D), r6i = r6 * idu, dlww = dl * ww;
  const T swe = r6i * See;  // r6 See / du
  T S[3];
  for (int i = 0; i < 3; ++i) S[i] = a[0][i] * mu[0] + a[1][i] * mu[1];
  // ---- F, and b = h F + ...
  T bx[2][3], be[2], re[2], Dm[2];
  for (int b = 0; b < 2; ++b) {
    Dm[b] = dot3(D, m[b]);
    re[b] = r6 * (2.0 * wD * mu[b] - dlww * mu[b] - Dm[b]);
  }
  {
    T rl = (s.over ? 4.0 * P.R : 2.0 * P.R) - du;
    if (rl < 0) rl = 0.0;
    const T crowd = P.kc * P.L * rl;
    const T Saa = dot3(a[0], m[0]) + dot3(a[1], m[1]);
    // stretch, gravity, contact and inertia act oppositely on the two ends
    const T Fe = 0.5 * (rho * gx - ks * (ww - 1.0) + r6 * (ww * See - Saa)) + crowd;
    const T F0 = Fe - re[0], F1 = -Fe - re[1];
    put(kE_fe + 0, in[0] ? F0 : zero);
    put(kE_fe + 1, in[1] ? F1 : zero);
    be[0] = h * F0;
    be[1] = h * F1;
    const T hr = 0.5 * (rho * du);
    for (int i = 0; i < 3; ++i) {
      const T t = strf * d[i] + r6 * (S[i] - See * w[i]), g = hr * P.G[i];
      bx[0][i] = h * (t - g - r6 * (dl * m[0][i] - mu[0] * D[i]));
      bx[1][i] = h * (-t - g - r6 * (dl * m[1][i] - mu[1] * D[i]));
    }
    // the Eulerian diagonal blocks: K_ee and D_ee
    const T Kee = ksi * ww;  // stretch: s (-ks ww / du)
    T kk[2][2], dd[2][2];
    for (int p = 0; p < 4; ++p) {
      const int ra = p >> 1, cb = p & 1;
      const T kin = r6i * (Dm[ra] - 3.0 * (dl * dot3(w, m[ra])) + 8.0 * (dlww * mu[ra]));
      const T base = ra == cb ? swe * ww - Kee : Kee - swe * ww;
      kk[ra][cb] = base - crowd + (cb == 0 ? -kin : kin) - r6 * re[ra];
    }
    dd[0][0] = dd[1][1] = (2.0 * r6) * (dlww - 2.0 * wD);
    dd[0][1] = (2.0 * r6) * (ww * mu[1] - wD);
    dd[1][0] = (-2.0 * r6) * (ww * mu[0] + wD);
    const T qw = q * ww;
    for (int p = 0; p < 4; ++p) {
      const int ra = p >> 1, cb = p & 1;
      const bool ok = ra == cb ? in[ra] : both;
      const T ee = (ra == cb ? 2.0 : 1.0) * qw + mh2 * kk[ra][cb] - h * dd[ra][cb];
      put(kE_ee + p, ok ? ee : zero);
      if (ra == cb) {
        put(kE_kee + ra, ok ? kk[ra][ra] : zero);
        put(kE_dee + ra, ok ? dd[ra][ra] : zero);
      }
    }
  }
  // ---- iso blocks
  {
    const T kI = mh2 * (swe * idu - ksi), hr6 = 2.0 * h * r6;
    put(kE_llI + 0, 2.0 * q + kI + hr6 * dl);
    put(kE_llI + 1, q - kI - hr6 * mu[0]);
    put(kE_llI + 2, q - kI + hr6 * mu[1]);
    put(kE_llI + 3, 2.0 * q + kI + hr6 * dl);
  }
  // ---- (M - h D^T) V, V = (a0, E0, a1, E1) with the interior velocities only.
  // M and D enter b without a graph in the reference (src/MatrixMp.cpp:40-99),
  // so the reference-mode tangents hold their factors constant.
  {
    auto cst = [&](const T& x) { return trunc ? detach(x) : x; };
    const T cq = cst(q), ce0 = cst(e[0]), ce1 = cst(e[1]), c2 = cst(-2.0 * h * r6);
    const T cm0 = 2.0 * ce0 + ce1, cm1 = ce0 + 2.0 * ce1, cdl = ce1 - ce0;
    T ca[2][3], cw[3], cD[3];
    for (int i = 0; i < 3; ++i) {
      ca[0][i] = cst(a[0][i]);
      ca[1][i] = cst(a[1][i]);
      cw[i] = cst(w[i]);
      cD[i] = ca[1][i] - ca[0][i];
    }
    const T E0 = in[0] ? e[0] : zero, E1 = in[1] ? e[1] : zero;
    const T B0 = both ? e[0] : zero, B1 = both ? e[1] : zero;
    // x rows: M, then -h D^T (c2 = -2 h r6)
    const T k0 = c2 * (E0 * cm0 + B1 * cm1) - cq * (2.0 * E0 + B1);
    const T k1 = -(c2 * (B0 * cm0 + E1 * cm1)) - cq * (2.0 * E1 + B0);
    const T x00 = 2.0 * cq - c2 * cdl, x01 = cq - c2 * cm1, x10 = cq + c2 * cm0;
    for (int i = 0; i < 3; ++i) {
      bx[0][i] += x00 * a[0][i] + x01 * a[1][i] + k0 * cw[i] - (3.0 * c2) * (E0 * ca[0][i]);
      bx[1][i] += x10 * a[0][i] + x00 * a[1][i] + k1 * cw[i] + (3.0 * c2) * (E1 * ca[1][i]);
    }
    // e rows
    const T wa0 = dot3(cw, a[0]), wa1 = dot3(cw, a[1]);
    const T cww = dot3(cw, cw), cwD = dot3(cw, cD);
    const T Da0 = dot3(cD, a[0]), Da1 = dot3(cD, a[1]);
    const T aa0 = dot3(ca[0], a[0]) + 2.0 * dot3(ca[1], a[0]), aa1 = 2.0 * dot3(ca[0], a[1]) + dot3(ca[1], a[1]);
    const T dia = cdl * cww - 2.0 * cwD;
    T r0 = c2 * (aa0 - cm0 * wa0 + dia * E0) - cq * (2.0 * wa0 - 2.0 * cww * E0);
    T r1 = c2 * (cm1 * wa1 - aa1 + dia * E1) - cq * (2.0 * wa1 - 2.0 * cww * E1);
    const T s0 = c2 * (Da1 + cm0 * wa1 - (cww * cm0 + cwD) * e[1]) - cq * (wa1 - cww * e[1]);
    const T s1 = c2 * (Da0 - cm1 * wa0 + (cww * cm1 - cwD) * e[0]) - cq * (wa0 - cww * e[0]);
    if (both) { r0 += s0; r1 += s1; }
    be[0] += r0;
    be[1] += r1;
    for (int i = 0; i < 3; ++i) { put(kE_b + i, bx[0][i]); put(kE_b + 4 + i, bx[1][i]); }
    put(kE_b + 3, in[0] ? be[0] : zero);
    put(kE_b + 7, in[1] ? be[1] : zero);
  }
  // ---- the mixed blocks, component by component
  {
    const T hr6 = -2.0 * h * r6;             // -h D's common factor
    const T p0 = mh2 * (r6i * mu[0]), p1 = mh2 * (r6i * mu[1]);
    const T kS = mh2 * r6i, kr = mh2 * (r6 * r6);
    const T uE = mh2 * (ksw - swe), uL = mh2 * (ksi + 3.0 * swe);
    const T q2 = -2.0 * q, hm0 = hr6 * mu[0], hm1 = hr6 * mu[1];
    for (int i = 0; i < 3; ++i) {
      const T g = (0.5 * mh2 * P.G[i]) * rho;
      const T sS = kS * S[i];
      const T U = uE * w[i] - sS, UL = uL * w[i] - sS;
      const T dw = dl * w[i];
      const T Y = D[i] - 3.0 * dw, Z = 2.0 * (D[i] - dw);
      const T R0 = kr * (dl * m[0][i] - mu[0] * D[i]), R1 = kr * (dl * m[1][i] - mu[1] * D[i]);
      const T y0 = p0 * Y - g, y1 = p1 * Y - g;
      // A[x(n_a)][e(n_c)] = -f q w - h^2 (s U + sw_c (mu_a Y - g) - r6 r_a) - h D
      const T le00 = (q2 - hm0) * w[i] + hr6 * m[1][i] + U - y0 - R0;
      const T le01 = (-q - hm1) * w[i] + hr6 * D[i] - U + y0 - R0;
      const T le10 = (hm0 - q) * w[i] + hr6 * D[i] - U - y1 - R1;
      const T le11 = (q2 + hm1) * w[i] - hr6 * m[0][i] + U + y1 - R1;
      // A[e(n_a)][x(n_c)] = -f q w - h^2 (s UL - sw_a g + sw_c mu_a Z) - h D
      const T z0 = p0 * Z, z1 = p1 * Z;
      const T el00 = (q2 + hm0) * w[i] - (3.0 * hr6) * a[0][i] + UL + g - z0;
      const T el01 = (-q - hm0) * w[i] - UL + g + z0;
      const T el10 = (hm1 - q) * w[i] - UL - g - z1;
      const T el11 = (q2 - hm1) * w[i] + (3.0 * hr6) * a[1][i] + UL - g + z1;
      put(kE_le + i, in[0] ? le00 : zero);
      put(kE_le + 3 + i, both ? le01 : zero);
      put(kE_le + 6 + i, both ? le10 : zero);
      put(kE_le + 9 + i, in[1] ? le11 : zero);
      put(kE_el + i, in[0] ? el00 : zero);
      put(kE_el + 3 + i, both ? el01 : zero);
      put(kE_el + 6 + i, both ? el10 : zero);
      put(kE_el + 9 + i, in[1] ? el11 : zero);
    }
  }
}
template <class T, class Put>
YS_HD void edge_terms(const View& v, int n0, int n1, int k, Put&& put) {
  edge_terms<T>(edge_load<T>(v, n0, n1, k), v.cp[v.node_cloth[n0]], k, v.h, v.trunc != 0, put);
}
template <class T>
YS_HD void edge_element(const View& v, int n0, int n1, int k, EdgeOut<T>& o) {
  edge_terms<T>(v, n0, n1, k, [&](int f, const T& x) { o.f[f] = x; });
}
// the record in the per-element buffer: field-major over the 2 * ntot edge
// slots (slot = k * ntot + n0), tangents in dbuf
template <class T>
YS_HD void edge_store(const View& v, double* buf, double* dbuf, int n0, int k, const EdgeOut<T>& o) {
  for (int f = 0; f < kEdgeFields; ++f) stT(buf, dbuf, 2 * f + k, v.ntot, n0, o.f[f]);
}

// ------------------------------------------------------------ bend element
// Geometry of a bend segment x2 - x0 - x1 and the factors of its terms
// (src/ClothUnit.h:197-210): unit directions d1, d2, a = P1 d2 and b = P2 d1
// (the directions projected across each other), the angle th of cosine
// c = -d1.d2 and 1 / sin(th). active is false for an exactly straight
// segment (sin = 0), where the reference switches bending off.
template <class T>
struct BendGeom {
  T il1, il2, d1[3], d2[3], a[3], b[3], th, c, is;
  bool active;
};
template <class T>
YS_HD void bend_geom(const T* to1, const T* to2, BendGeom<T>& g) {  // x1 - x0, x2 - x0
  for (int i = 0; i < 3; ++i) { g.d1[i] = to1[i]; g.d2[i] = to2[i]; }
  const T l1 = norm3(g.d1), l2 = norm3(g.d2);
  g.il1 = 1.0 / l1;
  g.il2 = 1.0 / l2;
  // rounded as divisions: a straight yarn along an axis has c = 1 exactly,
  // and with it no bending, where the reference has none
  for (int i = 0; i < 3; ++i) { g.d1[i] = quot(g.d1[i], l1, g.il1); g.d2[i] = quot(g.d2[i], l2, g.il2); }
  const T dd = dot3(g.d1, g.d2);
  for (int i = 0; i < 3; ++i) { g.a[i] = g.d2[i] - dd * g.d1[i]; g.b[i] = g.d1[i] - dd * g.d2[i]; }
  // the reference's clamp (EPS = DBL_MIN, src/Constants.h:25) acts only where
  // rounding has carried the cosine past +-1
  T c = -dd;
  if (c < -1.0) c = -1.0;
  if (c > 1.0) c = 1.0;
  g.c = c;
  g.th = acos(c);
  const T ss = (1.0 - c) * (1.0 + c);  // sin^2(th); zero exactly at c = +-1
  // a NaN counts as active, as sin(th) != 0 does
  g.active = !(ss == 0.0);
  g.is = g.active ? rsqrt_(ss) : T(0.0);
}

// Bend segment record (one per middle node and yarn direction), as it enters
// the system: the independent Hessian blocks scaled by -h^2 -- L11 and L22
// symmetric (xx, xy, xz, yy, yz, zz), L12 full, L21 its transpose (P1 P2 =
// (P2 P1)^T, and the rank-1 parts of src/PhysicsCloth.cpp:700-703 mirror each
// other) -- the forces F1, F2 of Bending_F, and those of the crimp segment
// that feed the compression estimate. The Eulerian couplings are
// L1E1 = -F1 / du, L2E1 = -F2 / du; the other blocks follow as in
// src/PhysicsCloth.cpp:705-727 and are formed by the gather. 37 fields for the
// 62 that hold every block: on 255,292 nodes the producer (FP64 bound) takes
// 0.33 ms for 0.63, the gather that reads the records 0.53 for 0.70.
constexpr int kB_L11 = 0, kB_L22 = 6, kB_L12 = 12, kB_F1 = 21, kB_F2 = 24, kB_idu = 27, kB_E1E1 = 28, kB_Fu2 = 29,
              kB_cF1 = 30, kB_cF2 = 33, kB_cidu = 36;
constexpr int kBendFields = 37;
YS_HD int sym3(int i, int j) { return i <= j ? i * (5 - i) / 2 + j : j * (5 - j) / 2 + i; }

// a diagonal block k (th (v d^T + cs2 v v^T + c (I - d d^T) + d v^T) - is v v^T)
template <class T, class Put>
YS_HD void bend_diag(const T& k, const T& th, const T& c, const T& kA, const T* vv, const T* d, int f, Put&& put) {
  const T kS = k * th, kP = kS * c;
  for (int i = 0; i < 3; ++i) {
    const T al = kA * vv[i] + kS * d[i], be = kS * vv[i] - kP * d[i];
    for (int j = i; j < 3; ++j) {
      const T x = al * vv[j] + be * d[j];
      put(f + sym3(i, j), i == j ? x + kP : x);
    }
  }
}

// Bending_F / Bending_D on the real nodes (src/PhysicsCloth.cpp:579-822) from
// the segment's arms x1 - x0 and x2 - x0, its Eulerian length and bending
// stiffness; put(field, value) receives its fields of the record once each.
template <class T, class Put>
YS_HD void bend_real(const T* to1, const T* to2, const T& du, const T& kb, double h, Put&& put) {
  BendGeom<T> g;
  bend_geom(to1, to2, g);
  const T idu = 1.0 / du;
  const T kt = kb * g.th * idu;
  put(kB_idu, idu);
  put(kB_Fu2, -kt * idu);
  put(kB_E1E1, (-2.0 * kt * g.th) * (idu * idu));
  const T on = g.active ? kb : T(0.0);
  const T f = -2.0 * (on * g.th) * (idu * g.is), f1 = f * g.il1, f2 = f * g.il2;
  for (int i = 0; i < 3; ++i) { put(kB_F1 + i, f1 * g.a[i]); put(kB_F2 + i, f2 * g.b[i]); }
  const T K = (-2.0 * h * h) * on * (idu * g.is);  // 2 kb / (du sin), scaled by -h^2
  const T k11 = K * (g.il1 * g.il1), k22 = K * (g.il2 * g.il2), k12 = -K * (g.il1 * g.il2);
  const T tc = g.th * (g.c * (g.is * g.is)) - g.is;
  bend_diag(k11, g.th, g.c, k11 * tc, g.a, g.d1, kB_L11, put);
  bend_diag(k22, g.th, g.c, k22 * tc, g.b, g.d2, kB_L22, put);
  // L12 = k12 (th P1 P2 - tc a b^T), P1 P2 = I - d1 d1^T - a d2^T
  const T kt12 = k12 * g.th, kab = -k12 * tc;
  for (int j = 0; j < 3; ++j) {
    const T pa = kab * g.b[j] - kt12 * g.d2[j], pd = -kt12 * g.d1[j];
    for (int i = 0; i < 3; ++i) {
      const T x = pa * g.a[i] + pd * g.d1[i];
      put(kB_L12 + 3 * i + j, i == j ? x + kt12 : x);
    }
  }
}
// Crimp_Bending_F / Crimp_Bending_D (src/PhysicsCloth.cpp:824-987) from the
// arms of the crimp-offset centre line; icu: reciprocal of the Eulerian
// length of the build, which crimp segments keep (src/Cloth.cpp:107)
template <class T, class Put>
YS_HD void bend_crimp(const T* to1, const T* to2, double icu, const T& kb, Put&& put) {
  BendGeom<T> g;
  bend_geom(to1, to2, g);
  const T f = g.active ? T((-2.0 * icu) * (kb * g.th) * g.is) : T(0.0), f1 = f * g.il1, f2 = f * g.il2;
  put(kB_cidu, T(icu));
  for (int i = 0; i < 3; ++i) { put(kB_cF1 + i, f1 * g.a[i]); put(kB_cF2 + i, f2 * g.b[i]); }
}
// the crimp-offset position of node n: x - R n along the warp, x + R n along the weft
template <class T>
YS_HD void crimp_point(const View& v, int n, int k, T* x) {
  const double R = v.cp[v.node_cloth[n]].R, sg = k == 0 ? -R : R;
  const bool in = (v.flags[n] & YS_INTERIOR) != 0;
  for (int i = 0; i < 3; ++i) {
    x[i] = ldT<T>(v.X, v.dX, i, v.ntot, n);
    if (in) x[i] += sg * ldT<T>(v.NRM, v.dNRM, i, v.ntot, n);
  }
}
YS_HD double crimp_icu(const View& v, int n2, int n1, int k) {
  return 1.0 / (ld(v.UV0, k, v.ntot, n1) - ld(v.UV0, k, v.ntot, n2));
}
// both for the segment n2 - n0 - n1 along yarn direction k
template <class T, class Put>
YS_HD void bend_terms(const View& v, int n2, int n0, int n1, int k, int line, Put&& put) {
  const int nt = v.ntot;
  const T kb = ldpT<T>(v.line_kb, v.dline_kb, line, v.nlines);
  T to1[3], to2[3];
  for (int i = 0; i < 3; ++i) {
    const T x0 = ldT<T>(v.X, v.dX, i, nt, n0);
    to1[i] = ldT<T>(v.X, v.dX, i, nt, n1) - x0;
    to2[i] = ldT<T>(v.X, v.dX, i, nt, n2) - x0;
  }
  bend_real(to1, to2, ldT<T>(v.UV, v.dUV, k, nt, n1) - ldT<T>(v.UV, v.dUV, k, nt, n2), kb, v.h, put);
  T x0[3];
  crimp_point(v, n0, k, x0);
  crimp_point(v, n1, k, to1);
  crimp_point(v, n2, k, to2);
  for (int i = 0; i < 3; ++i) { to1[i] -= x0[i]; to2[i] -= x0[i]; }
  bend_crimp(to1, to2, crimp_icu(v, n2, n1, k), kb, put);
}
// the record in the bend buffer at slot k * ntot + n0
template <class T>
YS_HD void bend_element(const View& v, double* buf, double* dbuf, int n2, int n0, int n1, int k, int line) {
  bend_terms<T>(v, n2, n0, n1, k, line, [&](int f, const T& x) { stT(buf, dbuf, 2 * f + k, v.ntot, n0, x); });
}

// ------------------------------------------------------------ wind (faces)
// Wind_F (src/PhysicsCloth.cpp:3091-3107), face geometry src/ClothUnit.h:268-273,
// from the face's edges e1, e2 and the sum of its nodes' velocities; f3 =
// wind_force / 3, the share of each of its three nodes. area n = cr / 2 and
// area tang = |cr| rel / 2 - vn cr / 2, so one division serves what nine
// did (FP64 divisions bound the kernel: 59 us for 203 on 255,292 nodes).
template <class T>
YS_HD void wind_terms(const ClothParams& P, const T* e1, const T* e2, const T* vs, T* f3) {
  T cr[3], rel[3];
  cross3(e1, e2, cr);
  const T cc = dot3(cr, cr);
  const T nc = sqrt(cc), inc = cc == 0.0 ? T(0.0) : 1.0 / nc;  // |cr|, 1 / |cr| (0 for a flat face)
  for (int i = 0; i < 3; ++i) rel[i] = P.wind[i] - vs[i] * (1.0 / 3.0);
  const T vn = dot3(cr, rel) * inc;
  const T k = (1.0 / 6.0) * vn * (P.wind_rho * fabs(vn) - P.wind_drag);
  const T kd = (P.wind_drag / 6.0) * nc;
  for (int i = 0; i < 3; ++i) f3[i] = k * cr[i] + kd * rel[i];
}
template <class T>
YS_HD void wind_face(const View& v, const ClothParams& P, int n1, int n2, int n3, T* f3) {
  const int nt = v.ntot;
  T e1[3], e2[3], vs[3];
  for (int i = 0; i < 3; ++i) {
    const T xa = ldT<T>(v.X, v.dX, i, nt, n1);
    e1[i] = ldT<T>(v.X, v.dX, i, nt, n2) - xa;
    e2[i] = ldT<T>(v.X, v.dX, i, nt, n3) - xa;
    vs[i] = ldT<T>(v.V, v.dV, i, nt, n1) + ldT<T>(v.V, v.dV, i, nt, n2) + ldT<T>(v.V, v.dV, i, nt, n3);
  }
  wind_terms(P, e1, e2, vs, f3);
}
// the nodes of face `which` (0, 1) of the cell with top-left node tl
YS_HD void cell_face(const View& v, int tl, int which, int n[3]) {
  const int W = v.cp[v.node_cloth[tl]].W, tr = tl + 1, bl = tl + W, br = tl + W + 1;
  const bool even = ((v.node_u[tl] + v.node_v[tl]) & 1) == 0;
  n[0] = which == 0 || even ? tl : tr;
  n[1] = which == 0 ? tr : br;
  n[2] = which == 0 && even ? br : bl;
}

// cell with top-left node tl: faces (src/Cloth.cpp:271-287) written to the
// face buffer [6][ntot] (face A then face B, each wind_force / 3)
template <class T>
YS_HD void cell_faces(const View& v, double* buf, double* dbuf, int tl) {
  const ClothParams& P = v.cp[v.node_cloth[tl]];
  T fa[3], fb[3];
  int n[3];
  cell_face(v, tl, 0, n);
  wind_face(v, P, n[0], n[1], n[2], fa);
  cell_face(v, tl, 1, n);
  wind_face(v, P, n[0], n[1], n[2], fb);
  for (int i = 0; i < 3; ++i) {
    stT(buf, dbuf, i, v.ntot, tl, fa[i]);
    stT(buf, dbuf, 3 + i, v.ntot, tl, fb[i]);
  }
}

// ------------------------------------------------------------ crossing node
// Node normal (src/Cloth.cpp:440-463): smallest right singular vector of the
// centred 5-point stencil = eigenvector of the smallest eigenvalue of its 3x3
// scatter matrix (cyclic Jacobi rotations), signed by warp x weft and the
// weave's flip flag.
// a <- diagonalised S, V <- its eigenvectors (columns)
YS_HD void sym3_jacobi(const double S[3][3], double a[3][3], double V[3][3]) {
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) V[i][j] = i == j ? 1.0 : 0.0;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) a[i][j] = S[i][j];
  // off-diagonal entries below 1e-24 of the diagonal scale move the
  // eigenvectors by less than 1e-24 and are treated as zero
  const double tiny = 1e-24 * (fabs(S[0][0]) + fabs(S[1][1]) + fabs(S[2][2]));
  for (int sweep = 0; sweep < 50; ++sweep) {
    if (fabs(a[0][1]) + fabs(a[0][2]) + fabs(a[1][2]) <= tiny) break;
    for (int p = 0; p < 2; ++p)
      for (int q = p + 1; q < 3; ++q) {
        if (fabs(a[p][q]) <= tiny) continue;
        const double theta = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double cs = 1.0 / sqrt(t * t + 1.0), sn = t * cs;
        for (int k = 0; k < 3; ++k) {
          const double akp = a[k][p], akq = a[k][q];
          a[k][p] = cs * akp - sn * akq;
          a[k][q] = sn * akp + cs * akq;
        }
        for (int k = 0; k < 3; ++k) {
          const double apk = a[p][k], aqk = a[q][k];
          a[p][k] = cs * apk - sn * aqk;
          a[q][k] = sn * apk + cs * aqk;
        }
        for (int k = 0; k < 3; ++k) {
          const double vkp = V[k][p], vkq = V[k][q];
          V[k][p] = cs * vkp - sn * vkq;
          V[k][q] = sn * vkp + cs * vkq;
        }
      }
  }
}
YS_HD int sym3_argmin(const double a[3][3]) {
  int m = 0;
  if (a[1][1] < a[m][m]) m = 1;
  if (a[2][2] < a[m][m]) m = 2;
  return m;
}
YS_HD void sym3_min_eigvec(const double S[3][3], double* out) {
  double a[3][3], V[3][3];
  sym3_jacobi(S, a, V);
  const int m = sym3_argmin(a);
  for (int k = 0; k < 3; ++k) out[k] = V[k][m];
}

// One step of Rayleigh-quotient iteration on a symmetric 3x3 S: x <- adj(S - mu
// I) x / |.|, mu = x^T S x (the adjugate solves the shifted system up to scale
// without a division and stays exact when mu hits the eigenvalue); false where
// x is already exact. Converges cubically.
template <class F>
YS_HD bool rqi_step(const F S[3][3], F x[3]) {
  F Sx[3];
  for (int i = 0; i < 3; ++i) Sx[i] = S[i][0] * x[0] + S[i][1] * x[1] + S[i][2] * x[2];
  const F mu = x[0] * Sx[0] + x[1] * Sx[1] + x[2] * Sx[2];
  const F m00 = S[0][0] - mu, m11 = S[1][1] - mu, m22 = S[2][2] - mu;
  const F m01 = S[0][1], m02 = S[0][2], m12 = S[1][2];
  // adjugate of the symmetric M = S - mu I
  const F c00 = m11 * m22 - m12 * m12, c01 = m02 * m12 - m01 * m22, c02 = m01 * m12 - m02 * m11;
  const F c11 = m00 * m22 - m02 * m02, c12 = m01 * m02 - m00 * m12, c22 = m00 * m11 - m01 * m01;
  const F y[3] = {c00 * x[0] + c01 * x[1] + c02 * x[2], c01 * x[0] + c11 * x[1] + c12 * x[2],
                  c02 * x[0] + c12 * x[1] + c22 * x[2]};
  const F ny = sqrt(y[0] * y[0] + y[1] * y[1] + y[2] * y[2]);
  if (!(ny > F(0)) || !isfinite(ny)) return false;
  const F iy = F(1) / ny;
  for (int i = 0; i < 3; ++i) x[i] = y[i] * iy;
  return true;
}

// Eigenvector of the smallest eigenvalue of a symmetric 3x3 S by Rayleigh-
// quotient iteration from a guess close to it. Returns false (out untouched)
// unless the result is an eigenvector of the smallest eigenvalue to 1e-15
// relative, for the caller to fall back on the Jacobi solver. Bound by the FP64
// pipe: three steps in FP32 (on S scaled to trace 1) bring the guess to 1e-6,
// from where FP64 steps go on: a second one unless the first left a residual
// below a sixth of a rounding of S (it does on smooth cloths), and up to two more
// on crumpled ones. Over random stencils (400,000 each) the error against
// extended precision is that of four FP64 steps from the guess or less (the
// largest 5.7e-17 for 7.2e-17, 1.35e-16 for 1.29e-16 and 2.2e-16 for 2e-11 where
// the crossings lie 0.05, 0.1 and 0.2 spacings out of place; the mean within 2 %).
// 255,292 normals take 133 us, 191 with four FP64 steps from the guess, 109 with
// one step where a residual of nine roundings sufficed; one 50 x 50 cloth 18, 22
// and 16.
YS_HD bool sym3_min_eigvec_rqi(const double S[3][3], const double* guess, double* out) {
  const double tr = S[0][0] + S[1][1] + S[2][2];
  double x[3];
  {
    const float gs = (float)fmax(fabs(guess[0]), fmax(fabs(guess[1]), fabs(guess[2])));
    float Sf[3][3], xf[3];
    const float ts = 1.0f / (float)tr, g1 = 1.0f / gs;
    bool ok = gs > 0.0f && isfinite(g1) && isfinite(ts) && ts > 0.0f;
    for (int i = 0; i < 3; ++i) {
      xf[i] = (float)guess[i] * g1;
      for (int j = 0; j < 3; ++j) Sf[i][j] = (float)S[i][j] * ts;
    }
    const float in = 1.0f / sqrt(xf[0] * xf[0] + xf[1] * xf[1] + xf[2] * xf[2]);
    for (int i = 0; i < 3; ++i) xf[i] *= in;
    for (int it = 0; it < 3 && ok; ++it)
      if (!rqi_step(Sf, xf)) break;
    const float n2 = xf[0] * xf[0] + xf[1] * xf[1] + xf[2] * xf[2];
    ok = ok && n2 > 0.5f && n2 < 2.0f;
    if (ok) {
      for (int i = 0; i < 3; ++i) x[i] = xf[i];
    } else {  // out of FP32's range
      const double nx = norm3(guess);
      if (!(nx > 0.0)) return false;
      for (int i = 0; i < 3; ++i) x[i] = guess[i] / nx;
    }
  }
  const double sc = fabs(S[0][0]) + fabs(S[1][1]) + fabs(S[2][2]) + 1e-300;
  double mu = 0.0, r2 = 0.0;
  for (int it = 0; it < 4; ++it) {
    const bool more = rqi_step(S, x);
    double Sx[3];
    for (int i = 0; i < 3; ++i) Sx[i] = S[i][0] * x[0] + S[i][1] * x[1] + S[i][2] * x[2];
    mu = dot3(x, Sx);
    r2 = 0.0;
    for (int i = 0; i < 3; ++i) r2 += (Sx[i] - mu * x[i]) * (Sx[i] - mu * x[i]);
    if (!more || r2 <= (it == 0 ? 3e-34 : 1e-30) * sc * sc) break;
  }
  if (!(r2 <= 1e-30 * sc * sc)) return false;
  // mu is the smallest eigenvalue iff the other two, l2 + l3 = tr - mu and
  // l2 l3 = e2 - mu (tr - mu), are both >= mu
  const double e2 = S[0][0] * S[1][1] + S[0][0] * S[2][2] + S[1][1] * S[2][2] - S[0][1] * S[0][1] -
                    S[0][2] * S[0][2] - S[1][2] * S[1][2];
  const double sum = tr - mu, prod = e2 - mu * sum;
  if (!(sum >= 2.0 * mu && prod - mu * sum + mu * mu >= -1e-12 * sc * sc)) return false;
  for (int i = 0; i < 3; ++i) out[i] = x[i];
  return true;
}

YS_HD void node_normal(const View& v, int n, int W) {
  const int nt = v.ntot;
  const int ids[5] = {n, n - 1, n + 1, n - W, n + W};
  double p[5][3], mean[3] = {0, 0, 0}, S[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  for (int m = 0; m < 5; ++m)
    for (int i = 0; i < 3; ++i) { p[m][i] = ld(v.X, i, nt, ids[m]); mean[i] += p[m][i]; }
  for (int i = 0; i < 3; ++i) mean[i] /= 5.0;
  for (int m = 0; m < 5; ++m) {
    double r[3] = {p[m][0] - mean[0], p[m][1] - mean[1], p[m][2] - mean[2]};
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) S[i][j] += r[i] * r[j];
  }
  double vw[3], vf[3], cr[3];
  for (int i = 0; i < 3; ++i) { vw[i] = p[2][i] - p[1][i]; vf[i] = p[4][i] - p[3][i]; }
  cross3(vw, vf, cr);
  // the smallest right singular vector of the centred positions (the
  // reference's torch::svd, src/Cloth.cpp:440-463) is the smallest
  // eigenvector of their scatter S; warp x weft is a close starting guess
  double nn[3];
  if (!sym3_min_eigvec_rqi(S, cr, nn)) sym3_min_eigvec(S, nn);
  const double len = norm3(nn), il = 1.0 / len;
  for (int i = 0; i < 3; ++i) nn[i] = quot(nn[i], len, il);
  const bool flip = (dot3(cr, nn) < 0) != ((v.flags[n] & YS_FLIP) != 0);
  for (int i = 0; i < 3; ++i) st(v.NRM, i, nt, n) = flip ? -nn[i] : nn[i];
}

// How the unit eigenvector n of a scatter matrix's smallest eigenvalue l_m moves:
// respond(r) = sum_{j != m} (v_j . r) / (l_m - l_j) v_j, the change of n for
// dS n = r (and its transpose). That is -M^-1 of r's part across n with M = S -
// l_m I + tr(S) n n^T, which needs no other eigenvector: one 3x3 inverse by
// cofactors where the eigensystem took a chain of some 20 rotations, 44 us of
// latency a launch.
struct NormalResponse {
  double n[3], c[6];  // the inverse's xx, xy, xz, yy, yz, zz
  YS_HD NormalResponse(const double S[3][3], const double* nn) {
    double Sn[3], mu = 0.0, m[6];
    for (int i = 0; i < 3; ++i) {
      n[i] = nn[i];
      Sn[i] = S[i][0] * nn[0] + S[i][1] * nn[1] + S[i][2] * nn[2];
    }
    for (int i = 0; i < 3; ++i) mu += nn[i] * Sn[i];
    const double tr = S[0][0] + S[1][1] + S[2][2];
    int k = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = i; j < 3; ++j, ++k) m[k] = S[i][j] + tr * (nn[i] * nn[j]) - (i == j ? mu : 0.0);
    c[0] = m[3] * m[5] - m[4] * m[4];
    c[1] = m[2] * m[4] - m[1] * m[5];
    c[2] = m[1] * m[4] - m[2] * m[3];
    c[3] = m[0] * m[5] - m[2] * m[2];
    c[4] = m[1] * m[2] - m[0] * m[4];
    c[5] = m[0] * m[3] - m[1] * m[1];
    const double id = -1.0 / (m[0] * c[0] + m[1] * c[1] + m[2] * c[2]);
    for (k = 0; k < 6; ++k) c[k] *= id;
  }
  YS_HD void respond(const double* r, double* g) const {
    const double a = n[0] * r[0] + n[1] * r[1] + n[2] * r[2];
    const double x = r[0] - a * n[0], y = r[1] - a * n[1], z = r[2] - a * n[2];
    g[0] = c[0] * x + c[1] * y + c[2] * z;
    g[1] = c[1] * x + c[3] * y + c[4] * z;
    g[2] = c[2] * x + c[4] * y + c[5] * z;
  }
};

// node_normal with tangents: the value as above; the tangent of the unit
// eigenvector n of the smallest eigenvalue l_m of the scatter S along dS is
// sum_{j != m} (v_j . dS n) / (l_m - l_j) v_j (first-order perturbation of a
// symmetric eigenproblem with simple eigenvalues, the derivative autograd
// takes through the SVD of src/Cloth.cpp:446). Values go to NRM, tangents
// to dNRM.
template <int K>
YS_HD void node_normal_dual(const View& v, int n, int W) {
  typedef Dual<K> D;
  const int nt = v.ntot;
  const int ids[5] = {n, n - 1, n + 1, n - W, n + W};
  D p[5][3], mean[3], S[3][3];
  for (int m = 0; m < 5; ++m)
    for (int i = 0; i < 3; ++i) { p[m][i] = ldT<D>(v.X, v.dX, i, nt, ids[m]); mean[i] += p[m][i]; }
  for (int i = 0; i < 3; ++i) mean[i] /= 5.0;
  for (int m = 0; m < 5; ++m) {
    D r[3] = {p[m][0] - mean[0], p[m][1] - mean[1], p[m][2] - mean[2]};
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) S[i][j] += r[i] * r[j];
  }
  double Sv[3][3], a[3][3], V[3][3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) Sv[i][j] = S[i][j].v;
  sym3_jacobi(Sv, a, V);
  const int mm = sym3_argmin(a);
  D nn[3];
  for (int i = 0; i < 3; ++i) nn[i] = D(V[i][mm]);
  for (int jj = 0; jj < 3; ++jj) {
    if (jj == mm) continue;
    const double gap = a[mm][mm] - a[jj][jj];
    for (int k = 0; k < K; ++k) {
      double c = 0.0;  // v_j . dS_k n
      for (int r = 0; r < 3; ++r)
        for (int q = 0; q < 3; ++q) c += V[r][jj] * S[r][q].d[k] * V[q][mm];
      for (int i = 0; i < 3; ++i) nn[i].d[k] += (c / gap) * V[i][jj];
    }
  }
  const D len = norm3(nn);
  for (int i = 0; i < 3; ++i) nn[i] /= len;
  double vw[3], vf[3], cr[3], nv[3];
  for (int i = 0; i < 3; ++i) {
    vw[i] = p[2][i].v - p[1][i].v;
    vf[i] = p[4][i].v - p[3][i].v;
    nv[i] = nn[i].v;
  }
  cross3(vw, vf, cr);
  if (dot3(cr, nv) / (norm3(cr) * norm3(nv)) < 0)
    for (int i = 0; i < 3; ++i) nn[i] = -nn[i];
  if (v.flags[n] & YS_FLIP)
    for (int i = 0; i < 3; ++i) nn[i] = -nn[i];
  for (int i = 0; i < 3; ++i) stT(v.NRM, v.dNRM, i, nt, n, nn[i]);
}

// The compression of crossing n from the summed crimp forces (src/PhysicsCloth.cpp:97-110)
template <class T>
YS_HD T crossing_comp(const View& v, int n, const T* cl) {
  T c = 0.0;
  for (int i = 0; i < 3; ++i) c += ldT<T>(v.NRM, v.dNRM, i, v.ntot, n) * cl[i];
  c *= 0.5;
  if (c < 0) c = 0.0;
  return c;
}

// ConSlideFriction (src/PhysicsCloth.cpp:2579-2641) for interior node n and
// yarn k from its gathered no-slide force FEns, its dF_E/dE diagonals EEp /
// EEv, the crossing's compression and that one's derivative sums cle; returns
// the A and b contributions of the E row and stores SLIDE.
template <class T>
YS_HD void friction_terms(const ClothParams& P, double h, bool trunc, const T& comp, const T& ce, const T& mu,
                          const T& uvm, const T& uvdot, const T& FEns, const T& EEp, const T& EEv, T& slide, T& aEE,
                          T& bE) {
  const double kf = P.kf, df = P.df, h2 = h * h;
  const T lim = comp * mu;
  slide = 1.0 / (1.0 + exp(-(1e4 * (fabs(FEns) - lim))));
  const T t = tanh(10 * uvm), tl = tanh(10 * (lim - FEns));
  const T ku = kf * uvm, tm = t * lim, mce = mu * ce;
  const T lo = -0.5 * (ku - tm);
  const T force = lo * tl + 0.5 * (ku + tm) - df * uvdot;
  const T g = (1.0 - t * t) * lim + t * mce;
  const T pos = -0.5 * (kf - g) * tl + lo * (1.0 - tl * tl) * (EEp - mce) - 0.5 * (kf + g);
  // tanh(10 * fric_lim - F) as written at src/PhysicsCloth.cpp:2630-2631
  const T tq = tanh(10 * lim - FEns);
  const T vel = lo * (1.0 - tq * tq) * EEv - df;
  aEE = -h2 * pos - h * vel;
  // D enters b without a graph in the reference (src/MatrixMp.cpp:40-99)
  bE = h * (force - (trunc ? detach(vel) : vel) * uvdot);
}
template <class T>
YS_HD void friction_node(const View& v, int n, int k, const T& comp, const T& FEns, const T& EEp, const T& EEv,
                         const T* cle, T& aEE, T& bE) {
  const int nt = v.ntot, c = v.node_cloth[n];
  T ce = 0.0, slide;
  for (int i = 0; i < 3; ++i) ce += ldT<T>(v.NRM, v.dNRM, i, nt, n) * cle[i];
  ce *= 0.5;
  const T uvm = ldT<T>(v.UV, v.dUV, k, nt, n) - ldT<T>(v.UVB, v.dUVB, k, nt, n);
  friction_terms(v.cp[c], v.h, v.trunc != 0, comp, ce, cloth_mu<T>(v, c), uvm, ldT<T>(v.UVD, v.dUVD, k, nt, n), FEns,
                 EEp, EEv, slide, aEE, bE);
  stT(v.SLIDE, v.dSLIDE, k, nt, n, slide);
}

// ------------------------------------------------------------ shear
// Shear segment record (one per crossing and segment type): the forces on the
// warp and weft neighbours scaled by h, and the four independent Hessian
// blocks as they enter A, scaled by -h^2 and transposed (To_Sparse_Mat,
// src/MatrixMp.cpp:54-65); the crossing's own force and blocks follow from
// them (src/PhysicsCloth.cpp:2710, 3033-3037) and are formed by the gather.
constexpr int kShearFields = 42;
constexpr int kS_F1 = 0, kS_F3 = 3, kS_J11 = 6, kS_J13 = 15, kS_J31 = 24, kS_J33 = 33;
// segment types in the order of src/Cloth.cpp:178-181: (warp, weft) offsets
YS_HD int shear_du(int seg) { return seg < 2 ? -1 : 1; }
YS_HD int shear_dv(int seg) { return (seg & 1) ? -1 : 1; }

// kA v v^T + kS (v d^T + d v^T - co d d^T) + kS co I, plus one + g v in row r
template <class T, class Put>
YS_HD void shear_diag(const T& kA, const T& kS, const T& co, const T* vv, const T* d, bool lock, const T& one,
                      const T& g, int f, Put&& put) {
  const T kP = kS * co;
  for (int i = 0; i < 3; ++i) {
    const T al = kA * vv[i] + kS * d[i], be = kS * vv[i] - kP * d[i];
    for (int j = i; j < 3; ++j) {
      T x = al * vv[j] + be * d[j];
      if (i == j) x += kP;
      if (lock) {
        put(f + 3 * i + j, x + (one + g * vv[i]));
        if (i != j) put(f + 3 * j + i, x + (one + g * vv[j]));
      } else {
        put(f + 3 * i + j, x);
        if (i != j) put(f + 3 * j + i, x);
      }
    }
  }
}

// Shear_F / Shear_D (src/PhysicsCloth.cpp:2643-3089) for crossing n0 with warp
// neighbour n1 = n0 + (shear_du, 0) and weft neighbour n3 = n0 + (0, shear_dv);
// put(field, value) receives each field of the record once.
// FP64-pipe bound: projections as d - (d.d') d', one reciprocal each for the
// lengths and for the lock's denominator, and the vanishing P3 d3 block left
// out took the producer from 1.23 to 0.95 ms on 255,292 nodes (0.97 M segments).
// One segment's inputs: the arms n1 - n0 and n3 - n0, and (compression + 1) S R^2
template <class T>
struct ShearIn {
  T d1[3], d3[3], SR;
  bool jam;  // the crossing's neighbours lie on its other side
};
template <class T>
YS_HD ShearIn<T> shear_load(const View& v, int n0, int seg) {
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  const int n1 = n0 + shear_du(seg), n3 = n0 + shear_dv(seg) * P.W, nt = v.ntot;
  ShearIn<T> s;
  s.SR = (ldT<T>(v.COMP, v.dCOMP, 0, nt, n0) + 1.0) * (cloth_S<T>(v, v.node_cloth[n0]) * (P.R * P.R));
  for (int i = 0; i < 3; ++i) {
    const T x0 = ldT<T>(v.X, v.dX, i, nt, n0);
    s.d1[i] = ldT<T>(v.X, v.dX, i, nt, n1) - x0;
    s.d3[i] = ldT<T>(v.X, v.dX, i, nt, n3) - x0;
  }
  const bool f0 = (v.flags[n0] & YS_FLIP) != 0, f1 = (v.flags[n1] & YS_FLIP) != 0, f3 = (v.flags[n3] & YS_FLIP) != 0;
  s.jam = f0 != f1 && f0 != f3;
  return s;
}
template <class T, class Put>
YS_HD void shear_terms(const ShearIn<T>& s, const ClothParams& P, double h, bool trunc, Put&& put) {
  const double Lc = P.L, R = P.R, mh2 = -(h * h);
  const T& SR = s.SR;
  T d1[3], d3[3], a3[3], a1[3];
  for (int i = 0; i < 3; ++i) { d1[i] = s.d1[i]; d3[i] = s.d3[i]; }
  const T il1 = rsqrt_(dot3(d1, d1)), il3 = rsqrt_(dot3(d3, d3));
  for (int i = 0; i < 3; ++i) { d1[i] *= il1; d3[i] *= il3; }
  // the crossing angle phi in [0, pi] and 1 / sin(phi) from its cosine co;
  // a3 = P1 d3, a1 = P3 d1, P = I - d d^T
  const T co = dot3(d1, d3);
  for (int i = 0; i < 3; ++i) { a3[i] = d3[i] - co * d1[i]; a1[i] = d1[i] - co * d3[i]; }
  const T phi = acos(co);
  const T is = rsqrt_((1.0 - co) * (1.0 + co)), is2 = is * is, cs2 = co * is2;
  const T i11 = il1 * il1, i33 = il3 * il3, i13 = il1 * il3;
  if (!s.jam) {
    const T kL = SR * (kPi * Lc) * is;
    const T ph = phi - kPi / 2;
    // Shear_F takes phi.item() in (phi - PI/2) (src/PhysicsCloth.cpp:2720-2721):
    // that factor carries no derivative along the reference's gradient path
    const T phf = trunc ? detach(phi) - kPi / 2 : ph;
    const T cf = h * (kL * phf), cf1 = cf * il1, cf3 = cf * il3;
    for (int i = 0; i < 3; ++i) { put(kS_F1 + i, cf1 * a3[i]); put(kS_F3 + i, cf3 * a1[i]); }
    // src/PhysicsCloth.cpp:2715-2751 per block:
    //   J11 = k11 (ph (-a3 d1^T + cs2 a3 a3^T - co P1 - d1 a3^T) - a3 a3^T / s)
    //   J13 = k13 ph (cs2 - 1/s) (a3 d1^T) P3 = k13 ph (cs2 - 1/s) a3 a1^T, as a1 = P3 d1
    // (J33, J31 likewise with 1 <-> 3)
    const T k = mh2 * kL, kA = k * (ph * cs2 - is), kS = -k * ph, kx = i13 * (k * ph) * (cs2 - is);
    shear_diag(kA * i11, kS * i11, co, a3, d1, false, kA, kA, kS_J11, put);
    shear_diag(kA * i33, kS * i33, co, a1, d3, false, kA, kA, kS_J33, put);
    for (int i = 0; i < 3; ++i) {
      const T x = kx * a3[i];
      for (int j = 0; j < 3; ++j) {
        const T y = x * a1[j];  // J13[i][j] = J31[j][i]
        put(kS_J13 + 3 * j + i, y);
        put(kS_J31 + 3 * i + j, y);
      }
    }
  } else {
    // jamming: smooth shear lock (src/PhysicsCloth.cpp:2656-2713, 2753-3031).
    // Every first derivative in those expressions is a multiple of
    // phi_x = -P d / (l sin phi) -- phi_s_x = sigma phi_x, con_func_x_x =
    // mu phi_x, gamma_x = kappa phi_x -- except kx_x, whose "1 - cf^2 cfx"
    // broadcasts a scalar 1 and so equals beta0 (1,1,1) + beta1 phi_x. With
    // the scalars below each Hessian entry is a short combination of rank-1
    // products; the arithmetic is the reference's, regrouped.
    const double pb = kPi / 2, sig = 0.6, LR = Lc / R;
    const double pb5 = P.pb5, pb4 = P.pb4;
    // half-angle sine and cosine: sqrt((1 -+ c) / 2), both >= 0 for phi in [0, pi]
    const T sh = sqrt(0.5 * (1.0 - co)), ch = sqrt(0.5 * (1.0 + co));
    const T gamma = LR * (sqrt(2.0) - 2.0 * sh);
    const T kap = -LR * ch;                       // gamma_x = kap * phi_x
    const T Aq = phi - P.jam, Bq = phi - pb;
    const T AB = Aq * Bq, phs = phi * AB;
    const T sgm = AB + phi * (Aq + Bq);           // phi_s_x = sgm * phi_x
    const T omg = 2.0 * (Aq + Bq + phi);
    const T num = pb5 * Aq, den = phs * phs + pb4 * sig * sig;
    const T rden = 1.0 / den, rden2 = rden * rden;
    const T cf = tanh(num * rden);
    const T ps2 = 2.0 * (phs * sgm);
    const T muc = (pb5 * den - num * ps2) * rden2;  // con_func_x_x = muc * phi_x
    const T g2 = gamma * gamma, g3 = g2 * gamma, g3c = 1.0 - g3, cf1m = 1.0 - cf, cf2 = cf * cf, eX = 1.0 - cf2;
    const T base2 = 0.5 * SR;
    const T kL = (kPi * Lc) * base2 * ((1.0 + g3) + g3c * cf);
    const T beta0 = kPi * base2 * g3c;
    const T beta1 = kPi * base2 * (3.0 * g2 * kap * cf1m - g3c * cf2 * muc);
    const T LBq = Lc * Bq, hLB2 = 0.5 * LBq * Bq;
    {
      const T u = -h * hLB2 * beta0, t = h * (hLB2 * beta1 + kL * Bq) * is, t1 = t * il1, t3 = t * il3;
      for (int i = 0; i < 3; ++i) { put(kS_F1 + i, u + t1 * a3[i]); put(kS_F3 + i, u + t3 * a1[i]); }
    }
    // The Hessian entries of src/PhysicsCloth.cpp:2753-3031 are, for each
    // block, one fixed linear map (scalars below) applied to a few per-entry
    // quantities: pxx (phi_x_x), O = phi_xa phi_xb^T, Ob = its mirror, Rg
    // (the gamma_x_x remainder), fo (the kx-constant term), plus the scalar 1
    // broadcast by "1 - cf^2 cfx" (x1x1, x3x3 only) and kx_x's beta0 (1,1,1)
    // rows/columns. Those quantities are in turn combinations of a handful of
    // rank-1 matrices (a3 a3^T, a3 d1^T + d1 a3^T, P1, ...), so each block is
    // J = sum_k c_k B_k with c_k computed once per block.
    // J = cP*pxx + cO*O + cOb*Ob + cR*Rg + fo (+ cOne*1 + row/column terms)
    const T kG = 3.0 * g2 * cf1m, kO = kap * (6.0 * gamma * kap * cf1m - 6.0 * g2 * eX * muc);
    const T cfqm2 = -2.0 * cf * eX * (muc * muc);
    const T X4 = 2.0 * muc * ps2 * rden;
    const T tnp = 2.0 * (num * phs) * rden2, tns2 = 2.0 * (num * (sgm * sgm)) * rden2, cross = ps2 * pb5 * rden2;
    const T cnx_p = pb5 * rden - tnp * sgm, tom = tnp * omg;
    const T H = (h * h) * hLB2 * base2;  // -h^2 times -(L Bq^2 / 2) base
    const T Hg = H * g3c, Hx = Hg * eX, HG = H * kG * kap;
    const T LB2 = 2.0 * mh2 * LBq, kLs = mh2 * kL;
    const T hk = H * kO - LB2 * beta1;
    const T hR = 0.5 * LR * (H * kG) * sh;
    const T kq = kLs * (Bq * cs2 - is), kB = kLs * Bq;
    // x1x1 and x3x3: psx = sgm pxx + omg O, cfdd = cfqm2 O + 1 - cf^2 cfx;
    // x1x1: pxx = r11 (S - cs2 A + co P1), O = Ob = rho1 A, Rg = qR11 A,
    //       fo = kL r11 (-Bq S + kq A - Bq co P1); A = a3 a3^T, S = a3 d1^T + d1 a3^T;
    // x3x3: the same with (a1, d3, P3)
    {
      const T cP = HG - Hg * cf2 * cnx_p;
      const T cO = hk + Hg * (cf2 * (tns2 + tom + X4) + cfqm2);
      const T kA = is * (kq - cP * cs2) + is2 * (cO + hR), kS = (cP - kB) * is;
      const T g = LB2 * beta0 * is;
      shear_diag(kA * i11, kS * i11, co, a3, d1, true, Hg, g * il1, kS_J11, put);
      shear_diag(kA * i33, kS * i33, co, a1, d3, true, Hg, g * il3, kS_J33, put);
    }
    // x1x3 (psx = sgm pxx + omg (O + Ob) / 2) and x3x1 (psx = sgm pxx + omg O);
    // both: nx += cross (O - Ob), cfdd = cfqm2 Ob + (1 - cf^2) cfx.
    // x1x3: pxx = -r13 (cs2 A + M), O = rho13 A, Ob = rho13 B, Rg = qR13 A,
    //       fo = kL r13 (kq A + Bq M); A = a3 a1^T, B = a1 a3^T, M = P1 P3
    // x3x1: pxx = -r13 M^T (its outer(P3 d1, d3) P3, src/PhysicsCloth.cpp:2775-2777,
    //       is zero: P3 d3 = 0), O = rho13 A, Ob = rho13 B, Rg = qR13 A,
    //       fo = kL r13 (kq A + Bq M^T); A = a1 a3^T, B = a3 a1^T
    {
      const T cP = HG + Hx * cnx_p, ik = i13 * is, ik2 = i13 * is2;
      const T com = hk + hR + Hx * (cross - tns2 - X4);
      const T kM = (kB - cP) * ik;
      const T g = 0.5 * LB2 * beta0 * is, g1 = g * il1, g3_ = g * il3;
      {  // M = I - d1 d1^T - a3 d3^T
        const T kA = ik * (kq - cP * cs2) + ik2 * (com - 0.5 * Hx * tom);
        const T kb = ik2 * (Hg * cfqm2 - Hx * (0.5 * tom + cross));
        for (int j = 0; j < 3; ++j) {
          const T pa3 = kA * a1[j] - kM * d3[j] + g1, pa1 = kb * a3[j], pd = -kM * d1[j], p0 = g3_ * a1[j];
          for (int i = 0; i < 3; ++i) {
            const T x = pa3 * a3[i] + pa1 * a1[i] + pd * d1[i] + p0;
            put(kS_J13 + 3 * j + i, i == j ? x + kM : x);
          }
        }
      }
      {  // M^T = I - d3 d3^T - a1 d1^T
        const T kA = ik * kq + ik2 * (com - Hx * tom);
        const T kb = ik2 * (Hg * cfqm2 - Hx * cross);
        for (int j = 0; j < 3; ++j) {
          const T pa1 = kA * a3[j] - kM * d1[j] + g3_, pa3 = kb * a1[j], pd = -kM * d3[j], p0 = g1 * a3[j];
          for (int i = 0; i < 3; ++i) {
            const T x = pa1 * a1[i] + pa3 * a3[i] + pd * d3[i] + p0;
            put(kS_J31 + 3 * j + i, i == j ? x + kM : x);
          }
        }
      }
    }
  }
}
// the record in the shear buffer at slot seg * ntot + n0
template <class T>
YS_HD void shear_element(const View& v, double* buf, double* dbuf, int n0, int seg) {
  shear_terms<T>(shear_load<T>(v, n0, seg), v.cp[v.node_cloth[n0]], v.h, v.trunc != 0, [&](int f, const T& x) {
    stT(buf, dbuf, 4 * f + seg, v.ntot, n0, x);
  });
}

}  // namespace ys
