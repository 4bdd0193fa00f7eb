// ys_items.cuh -- per-node bodies of the step kernels that are not element
// terms: gathering the element records into a row block, the stencil SpMV row,
// and the state update. Kept separate from the launch code so one node's work
// is a plain function of (View, node).
#pragma once

#include <type_traits>

#include "ys_physics.cuh"

namespace ys {

// Per-element record buffers of one step (field-major, coalesced over the
// anchor node). Edges and bend segments have one slot per node and yarn
// direction (slot = k * ntot + anchor), faces one per cell (top-left node),
// shear segments four per crossing (slot = type * ntot + crossing).
struct Records {
  double* edge;   // [kEdgeFields][2][ntot] (kE_* offsets)
  double* bend;   // [kBendFields][2][ntot]
  double* face;   // [6][ntot]
  double* shear;  // [kShearFields][4][ntot]
  // tangents of the same records (forward-mode runs only; layout of ys_physics.cuh lds)
  double* dedge;
  double* dbend;
  double* dface;
  double* dshear;
};

YS_HD double rec(const double* buf, int field, int nslot, int slot_, int ntot, int node) {
  return buf[((int64_t)field * nslot + slot_) * ntot + node];
}
template <class T>
YS_HD T recT(const double* buf, const double* dbuf, int field, int nslot, int slot_, int ntot, int node) {
  return ldT<T>(buf, dbuf, field * nslot + slot_, ntot, node);
}

// one coefficient slot of row block n (value, and tangents when T is a Dual)
template <class T>
YS_HD void stA(const View& v, int s, int n, const T& x) { stT(v.A, v.dA, s, v.ntot, n, x); }
template <class T>
YS_HD T ldA(const View& v, int s, int n) { return ldT<T>(v.A, v.dA, s, v.ntot, n); }

// every bit pattern but infinities and NaN; an integer test, as a compare would
// take the FP64 pipe the producers and gathers wait for
YS_HD bool finite_(double x) {
#if defined(__CUDA_ARCH__)
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
#else
  return isfinite(x);
#endif
}

// The two gathers split a node's work into four parts, one per yarn neighbour
// m = 0..3: (-1, 0), (1, 0), (0, -1), (0, 1). Part m sums what the elements
// towards that neighbour give to the node's own block, and owns the blocks
// towards the neighbour, towards the next crossing beyond it and towards one
// diagonal neighbour. No record is read by two parts except a bend segment's
// L12 and forces (by the two parts along its yarn). On the device four warps
// run the parts of 32 nodes and combine the sums through shared memory, so a
// small cloth has four times the threads and a quarter of the chain; combined
// in the same order on the host.
YS_HD int part_k(int m) { return m >> 1; }
YS_HD int part_dir(int m) { return (m & 1) ? 1 : -1; }

struct NodeAt {
  int n, u, w, W, H;
  bool in;
  YS_HD NodeAt(const View& v, int n_) : n(n_) {
    const ClothParams& P = v.cp[v.node_cloth[n]];
    W = P.W;
    H = P.H;
    u = v.node_u[n];
    w = v.node_v[n];
    in = (v.flags[n] & YS_INTERIOR) != 0;
  }
  YS_HD int step(int k) const { return k == 0 ? 1 : W; }
  YS_HD int pos(int k) const { return k == 0 ? u : w; }
  YS_HD int len(int k) const { return k == 0 ? W : H; }
  YS_HD bool interior(int uu, int vv) const { return uu >= 1 && uu <= W - 2 && vv >= 1 && vv <= H - 2; }
};

// ---- the crossing pass: ConSlideFriction's inputs (src/PhysicsCloth.cpp:97-131)
template <class T>
struct CrossPart {
  T CL[3];             // crimp compression, summed over the four parts
  T FE, KEE, DEE;      // no-slide force and stiffness along yarn k, over its two parts
  T CLE[3];
};
template <class T>
YS_HD void cross_part(const View& v, const Records& R, const NodeAt& N, int m, CrossPart<T>& c) {
  const int nt = v.ntot, n = N.n, k = part_k(m), dir = part_dir(m), step = N.step(k), pos = N.pos(k), len = N.len(k);
  for (int r = 0; r < 3; ++r) c.CL[r] = c.CLE[r] = 0.0;
  c.FE = c.KEE = c.DEE = 0.0;
  const double sgn = k == 0 ? 1.0 : -1.0;
  if (pos + dir >= 0 && pos + dir < len) {  // the edge: n is its n0 when dir = +1
    const int a = dir > 0 ? 0 : 1, anc = dir > 0 ? n : n - step;
    auto E = [&](int f) { return recT<T>(R.edge, R.dedge, f, 2, k, nt, anc); };
    const T cl = E(kE_cl), cle = E(kE_cle);
    for (int r = 0; r < 3; ++r) {
      const T d = E(kE_d + r);
      c.CL[r] += dir > 0 ? cl * d : -(cl * d);
      c.CLE[r] += cle * d;
    }
    c.FE += E(kE_fe + a);
    c.KEE += E(kE_kee + a);
    c.DEE += E(kE_dee + a);
  }
  const int mid = pos + dir;
  if (mid >= 1 && mid <= len - 2) {  // the segment centred on the neighbour: n is its n2 (dir = +1) or n1
    auto Bf = [&](int f) { return recT<T>(R.bend, R.dbend, f, 2, k, nt, n + dir * step); };
    const double end = dir;
    const T cidu = (end * sgn) * Bf(kB_cidu);
    for (int r = 0; r < 3; ++r) {
      const T cF = Bf((dir > 0 ? kB_cF2 : kB_cF1) + r);
      c.CL[r] += sgn * cF;
      c.CLE[r] += cidu * cF;
    }
    c.KEE += Bf(kB_E1E1);
    c.FE += end * Bf(kB_Fu2);
  }
  if (dir > 0 && pos >= 1 && pos <= len - 2) {  // the segment centred on n
    auto Bf = [&](int f) { return recT<T>(R.bend, R.dbend, f, 2, k, nt, n); };
    for (int r = 0; r < 3; ++r) c.CL[r] -= sgn * (Bf(kB_cF1 + r) + Bf(kB_cF2 + r));
  }
}

// the crossing pass of node n: stores COMP and SLIDE, and leaves friction's
// share of the Eulerian rows in their diagonal slots and in b
template <class T>
YS_HD void gather_elements(const View& v, const Records& R, int n) {
  const NodeAt N(v, n);
  if (!N.in) return;
  CrossPart<T> c[4];
  for (int m = 0; m < 4; ++m) cross_part(v, R, N, m, c[m]);
  T CL[3];
  for (int r = 0; r < 3; ++r) CL[r] = (c[0].CL[r] + c[1].CL[r]) + (c[2].CL[r] + c[3].CL[r]);
  const T comp = crossing_comp(v, n, CL);
  stT(v.COMP, v.dCOMP, 0, v.ntot, n, comp);
  for (int k = 0; k < 2; ++k) {
    const CrossPart<T>&a = c[2 * k], &b = c[2 * k + 1];
    const T CLE[3] = {a.CLE[0] + b.CLE[0], a.CLE[1] + b.CLE[1], a.CLE[2] + b.CLE[2]};
    T aEE, bE;
    friction_node(v, n, k, comp, a.FE + b.FE, a.KEE + b.KEE, a.DEE + b.DEE, CLE, aEE, bE);
    stA(v, YS_SLOT_EE_SELF + k, n, aEE);
    stT(v.B, v.dB, 3 + k, v.ntot, n, bE);
  }
}

// ---- the row pass
// what part m gives to the node's own block: LL and b of the x rows (summed
// over the four parts), and the Eulerian couplings of yarn k (over its two)
template <class T>
struct RowPart {
  T LL[9], B[3], LE[3], EL[3], EE, Be;
};
// The diagonal neighbour (dx, dy) gets J13 from part (u, dx) and J31 from
// part (v, dy). Part 0 owns (-1, -1), part 1 (1, 1), part 2 (1, -1), part 3
// (-1, 1); each sends one share and receives one:
YS_HD int diag_from(int m) { return m == 0 ? 2 : m == 1 ? 3 : m == 2 ? 1 : 0; }
YS_HD int diag_slot(int m) { return m == 0 ? 9 : m == 1 ? 12 : m == 2 ? 10 : 11; }

// Part m of row block n: writes the blocks towards the yarn neighbour and the
// crossing beyond it, fills the sums of `o`, and hands its entries i of the
// diagonal blocks to share(mine, i, value): mine, of the one it owns, else of
// the one it sends. Node-node blocks are in the
// orientation of the dense matrix (src/MatrixMp.cpp:54-65). Clears fin if a
// value written is not finite.
template <class T, class Share>
YS_HD void row_part(const View& v, const Records& R, const NodeAt& N, int m, RowPart<T>& o, bool& fin, Share&& share) {
  const int nt = v.ntot, n = N.n, k = part_k(m), dir = part_dir(m), step = N.step(k), pos = N.pos(k), len = N.len(k);
  const double h = v.h, mh2 = -(v.h * v.h);
  T nLL[9], nLE[3], nEL[3], nEE = 0.0;
  for (int i = 0; i < 9; ++i) o.LL[i] = nLL[i] = 0.0;
  for (int i = 0; i < 3; ++i) o.B[i] = o.LE[i] = o.EL[i] = nLE[i] = nEL[i] = 0.0;
  o.EE = o.Be = 0.0;
  const bool has = pos + dir >= 0 && pos + dir < len;
  const int nb = has ? n + dir * step : n;
  const bool inb = has && (v.flags[nb] & YS_INTERIOR) != 0;
  if (has) {  // the edge between n and nb
    const int a = dir > 0 ? 0 : 1, p = 3 * a, q = a + 1, anc = dir > 0 ? n : nb;
    auto E = [&](int f) { return recT<T>(R.edge, R.dedge, f, 2, k, nt, anc); };
    const T cP = E(kE_lP), cI = E(kE_llI + p), cJ = E(kE_llI + q);
    const T d[3] = {E(kE_d), E(kE_d + 1), E(kE_d + 2)};
    for (int r = 0; r < 3; ++r) {
      const T pd = cP * d[r];
      for (int c = 0; c < 3; ++c) {
        const T x = (r == c ? cP : T(0.0)) - pd * d[c];
        o.LL[3 * r + c] = r == c ? x + cI : x;
        nLL[3 * r + c] = r == c ? cJ - x : -x;
      }
      o.B[r] = E(kE_b + 4 * a + r);
      o.LE[r] = E(kE_le + 3 * p + r);
      o.EL[r] = E(kE_el + 3 * p + r);
      nLE[r] = E(kE_le + 3 * q + r);
      nEL[r] = E(kE_el + 3 * q + r);
    }
    o.EE = E(kE_ee + p);
    nEE = E(kE_ee + q);
    o.Be = E(kE_b + 4 * a + 3);
  }
  if (has && pos >= 1 && pos <= len - 2) {  // the bend segment centred on n (nb is its n1 if dir = +1, else n2)
    auto Bf = [&](int f) { return recT<T>(R.bend, R.dbend, f, 2, k, nt, n); };
    // L01 = -(L11 + L21), L02 = -(L12 + L22), written transposed; L21 = L12^T
    T own[6], x12[9], F[3];
    for (int i = 0; i < 6; ++i) own[i] = Bf((dir > 0 ? kB_L11 : kB_L22) + i);
    for (int i = 0; i < 9; ++i) x12[i] = Bf(kB_L12 + i);
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) nLL[3 * r + c] -= own[sym3(r, c)] + (dir > 0 ? x12[3 * r + c] : x12[3 * c + r]);
    for (int r = 0; r < 3; ++r) F[r] = Bf(kB_F1 + r) + Bf(kB_F2 + r);
    if (dir > 0) {  // the middle's own block L00 = L11 + L12 + L21 + L22 (src/PhysicsCloth.cpp:709); F_x0 = -(F_x1 + F_x2)
      for (int r = 0; r < 3; ++r) {
        for (int c = r; c < 3; ++c) {
          const T t = (own[sym3(r, c)] + Bf(kB_L22 + sym3(r, c))) + (x12[3 * r + c] + x12[3 * c + r]);
          o.LL[3 * r + c] += t;
          if (c != r) o.LL[3 * c + r] += t;
        }
        o.B[r] -= h * F[r];
      }
    }
    // Eulerian couplings of Bending_D (src/PhysicsCloth.cpp:774-822):
    // q = L1E1 + L2E1 = L0E2 = E2L0 = -L0E1 = -E1L0
    if (N.in && inb) {
      const T t = -mh2 * Bf(kB_idu);
      for (int r = 0; r < 3; ++r) {
        const T q = t * F[r];
        if (dir < 0) { nLE[r] += q; nEL[r] += q; }  // row n0, column e / x of n2
        else nLE[r] -= q;                           // row n0, column e of n1
      }
    }
  }
  const int mid = pos + dir;
  const bool beyond = mid >= 1 && mid <= len - 2;
  if (beyond) {  // the segment centred on nb: n is its n2 (dir = +1) or its n1
    auto Bf = [&](int f) { return recT<T>(R.bend, R.dbend, f, 2, k, nt, nb); };
    T own[6], x12[9], F[3], G[3];
    for (int i = 0; i < 6; ++i) own[i] = Bf((dir > 0 ? kB_L22 : kB_L11) + i);
    for (int i = 0; i < 9; ++i) x12[i] = Bf(kB_L12 + i);
    const int s2 = stencil_index(k == 0 ? 2 * dir : 0, k == 1 ? 2 * dir : 0);
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) {
        // L20 = -(L21 + L22) or L10 = -(L11 + L12), and L21 or L12, transposed
        const T x = dir > 0 ? x12[3 * r + c] : x12[3 * c + r], t = own[sym3(r, c)];
        o.LL[3 * r + c] += t;
        nLL[3 * r + c] -= t + x;
        fin = fin && finite_(val(x));
        stA(v, YS_SLOT_LL + 9 * s2 + 3 * r + c, n, x);
      }
    for (int r = 0; r < 3; ++r) {
      F[r] = Bf((dir > 0 ? kB_F2 : kB_F1) + r);
      G[r] = Bf((dir > 0 ? kB_F1 : kB_F2) + r);
      o.B[r] += h * F[r];
    }
    if (N.in) {  // n2 (src/PhysicsCloth.cpp:737-753) or n1 (755-772)
      const T t = mh2 * Bf(kB_idu);
      for (int r = 0; r < 3; ++r) {
        const T x = t * F[r];
        if (dir > 0) { o.LE[r] += x; o.EL[r] += x; }
        else { o.LE[r] -= x; o.EL[r] -= x; }
        if (dir < 0 && inb) nEL[r] += x + t * G[r];  // row n1, column x of n0
      }
      o.EE += mh2 * Bf(kB_E1E1);
      const T fu = h * Bf(kB_Fu2);
      o.Be += dir > 0 ? fu : -fu;
    }
  } else {
    const int s2 = stencil_index(k == 0 ? 2 * dir : 0, k == 1 ? 2 * dir : 0);
    for (int i = 0; i < 9; ++i) stA(v, YS_SLOT_LL + 9 * s2 + i, n, T(0.0));
  }
  {  // wind on the cell (u - 1 + (m & 1), v - 1 + (m >> 1)) (src/Cloth.cpp:271-287)
    const int ci = N.u - 1 + (m & 1), cj = N.w - 1 + (m >> 1);
    if (ci >= 0 && ci < N.W - 1 && cj >= 0 && cj < N.H - 1) {
      const int tl = n + (ci - N.u) + (cj - N.w) * N.W;
      const bool right = ci != N.u, below = cj != N.w;  // n is tr / bl / br of that cell
      const bool even = ((ci + cj) & 1) == 0;
      const bool inA = !below || right == even, inB = below || right != even;
      for (int r = 0; r < 3; ++r) {
        if (inA) o.B[r] += h * ldT<T>(R.face, R.dface, r, nt, tl);
        if (inB) o.B[r] += h * ldT<T>(R.face, R.dface, 3 + r, nt, tl);
      }
    }
  }
  // shear segments (src/PhysicsCloth.cpp:2643-3089, 3033-3047). For part
  // (u, dir): J11 / J13 / F1, and J31 towards the crossing; for part (v, dir)
  // the same with 1 <-> 3.
  const int f1 = k == 0 ? kS_J11 : kS_J33, f13 = k == 0 ? kS_J13 : kS_J31, f31 = k == 0 ? kS_J31 : kS_J13;
  const int fF = k == 0 ? kS_F1 : kS_F3;
  if (N.in) {  // n is the crossing: its two segments towards nb
    T t[9];
    for (int i = 0; i < 9; ++i) t[i] = 0.0;
    for (int j = 0; j < 2; ++j) {
      const int seg = k == 0 ? (dir > 0 ? 2 : 0) + j : 2 * j + (dir > 0 ? 0 : 1);
      for (int i = 0; i < 9; ++i)
        t[i] += recT<T>(R.shear, R.dshear, f1 + i, 4, seg, nt, n) + recT<T>(R.shear, R.dshear, f31 + i, 4, seg, nt, n);
      for (int r = 0; r < 3; ++r) o.B[r] -= recT<T>(R.shear, R.dshear, fF + r, 4, seg, nt, n);
    }
    for (int i = 0; i < 9; ++i) {  // J01 or J03 = -(J11 + J31), and its share of J00
      o.LL[i] += t[i];
      nLL[i] -= t[i];
    }
  }
  if (inb) {  // nb is the crossing, n the end of two of its segments (on its side -dir)
    for (int j = 0; j < 2; ++j) {
      const int seg = k == 0 ? (dir > 0 ? 0 : 2) + j : 2 * j + (dir > 0 ? 1 : 0);
      // the segment's other end lies at offset `side` across the yarn
      const int side = k == 0 ? shear_dv(seg) : shear_du(seg);
      const bool mine = k == 0 ? side == dir : side != dir;
      for (int i = 0; i < 9; ++i) {
        const T a = recT<T>(R.shear, R.dshear, f1 + i, 4, seg, nt, nb), b = recT<T>(R.shear, R.dshear, f13 + i, 4, seg, nt, nb);
        o.LL[i] += a;
        nLL[i] -= a + b;  // J10 or J30
        share(mine, i, b);
      }
      for (int r = 0; r < 3; ++r) o.B[r] += recT<T>(R.shear, R.dshear, fF + r, 4, seg, nt, nb);
    }
  } else {
    for (int i = 0; i < 9; ++i) {
      share(true, i, T(0.0));
      share(false, i, T(0.0));
    }
  }
  const int s1 = stencil_index(k == 0 ? dir : 0, k == 1 ? dir : 0);
  for (int i = 0; i < 9; ++i) {
    fin = fin && finite_(val(nLL[i]));
    stA(v, YS_SLOT_LL + 9 * s1 + i, n, nLL[i]);
  }
  for (int r = 0; r < 3; ++r) {
    fin = fin && finite_(val(nLE[r])) && finite_(val(nEL[r]));
    stA(v, YS_SLOT_LE_NBR + 3 * m + r, n, nLE[r]);
    stA(v, YS_SLOT_EL_NBR + 3 * m + r, n, nEL[r]);
  }
  fin = fin && finite_(val(nEE));
  stA(v, YS_SLOT_EE_NBR + m, n, nEE);
}

// Row r of the node's own block from the summed parts: the handle spring
// (Constraint_F / Constraint_D, src/PhysicsCloth.cpp:232-248), the external
// force of SimStep(..., ext_force) (src/TrainHelper.cpp:63) and the Jacobi
// preconditioner (zero diagonal -> 1, as Eigen's DiagonalPreconditioner)
template <class T>
YS_HD void row_self_x(const View& v, int n, int r, const T* LL3, T b, double* dinv, bool& fin) {
  const int nt = v.ntot;
  const double h = v.h;
  T dg = LL3[r];
  if (v.flags[n] & YS_FIXED) {
    const double kh = v.cp[v.node_cloth[n]].kh;
    b += h * (-(kh * (ldT<T>(v.X, v.dX, r, nt, n) - ld(v.XF, r, nt, n))));
    dg += (h * h) * kh;
  }
  if (v.ext) b += h * ld(v.ext, r, nt, n);
  for (int c = 0; c < 3; ++c) {
    const T x = c == r ? dg : LL3[c];
    fin = fin && finite_(val(x));
    stA(v, YS_SLOT_LL + 3 * r + c, n, x);
  }
  fin = fin && finite_(val(b));
  stT(v.B, v.dB, r, nt, n, b);
  if (dinv) st(dinv, r, nt, n) = val(dg) != 0.0 ? 1.0 / val(dg) : 1.0;
}
// the Eulerian row of yarn k (an identity row on the boundary), with the
// crossing pass's friction
template <class T>
YS_HD void row_self_e(const View& v, int n, int k, bool in, const T* LE, const T* EL, T ee, T b, double* dinv, bool& fin) {
  const int nt = v.ntot;
  if (in) {
    ee += ldA<T>(v, YS_SLOT_EE_SELF + k, n);
    b += ldT<T>(v.B, v.dB, 3 + k, nt, n);
    if (v.ext) b += v.h * ld(v.ext, 3 + k, nt, n);
  } else {
    ee = T(1.0);
    b = T(0.0);
  }
  for (int r = 0; r < 3; ++r) {
    fin = fin && finite_(val(LE[r])) && finite_(val(EL[r]));
    stA(v, YS_SLOT_LE_SELF + 2 * r + k, n, LE[r]);
    stA(v, YS_SLOT_EL_SELF + 3 * k + r, n, EL[r]);
  }
  fin = fin && finite_(val(ee)) && finite_(val(b));
  stA(v, YS_SLOT_EE_SELF + k, n, ee);
  stT(v.B, v.dB, 3 + k, nt, n, b);
  if (dinv) st(dinv, 3 + k, nt, n) = val(ee) != 0.0 ? 1.0 / val(ee) : 1.0;
}

// Row block n whole, after the crossing pass and the shear records: all 159
// slots and b. Returns false if it holds a non-finite value (SimStep's
// DetectNaN / DetectInf, src/TrainHelper.cpp:22-37).
template <class T>
YS_HD bool gather_shear_finalize(const View& v, const Records& R, int n, double* dinv) {
  const NodeAt N(v, n);
  bool fin = true;
  RowPart<T> o[4];
  T dg[2][4][9];
  for (int m = 0; m < 4; ++m)
    row_part(v, R, N, m, o[m], fin, [&](bool mine, int i, const T& x) { dg[mine ? 0 : 1][m][i] = x; });
  T LL[9];
  for (int i = 0; i < 9; ++i) LL[i] = (o[0].LL[i] + o[1].LL[i]) + (o[2].LL[i] + o[3].LL[i]);
  for (int r = 0; r < 3; ++r)
    row_self_x<T>(v, n, r, LL + 3 * r, (o[0].B[r] + o[1].B[r]) + (o[2].B[r] + o[3].B[r]), dinv, fin);
  for (int k = 0; k < 2; ++k) {
    const RowPart<T>&a = o[2 * k], &b = o[2 * k + 1];
    T LE[3], EL[3];
    for (int r = 0; r < 3; ++r) { LE[r] = a.LE[r] + b.LE[r]; EL[r] = a.EL[r] + b.EL[r]; }
    row_self_e<T>(v, n, k, N.in, LE, EL, a.EE + b.EE, a.Be + b.Be, dinv, fin);
  }
  for (int m = 0; m < 4; ++m)
    for (int i = 0; i < 9; ++i) {
      const T x = dg[0][m][i] + dg[1][diag_from(m)][i];
      fin = fin && finite_(val(x));
      stA(v, YS_SLOT_LL + 9 * diag_slot(m) + i, n, x);
    }
  return fin;
}

// The SpMV rows read their input vector through an accessor: at(j) is a
// handle of node j and get(p, c) its component c. The global form below
// reads a [5][ntot] array; the persistent PCG reads its direction from the
// shared memory of the CTAs of a cluster through another accessor. Both run
// the same arithmetic, so they give the same bits.
struct GlobalVec {
  const double* YS_RESTRICT x;
  int64_t nt;
  typedef const double* Ptr;
  YS_HD Ptr at(int j) const { return x + j; }
  YS_HD double get(Ptr p, int c) const { return p[c * nt]; }
};

// y = A x for row block n (5 rows). Couplings to grid positions outside the
// cloth have zero coefficients; their column index is clamped to n so the
// load stays in bounds and adds 0 * x(n). Every coefficient enters one fused
// multiply-add into its row's running sum, in slot order: 159 FMAs a row
// block, the FP64 pipe's floor for this product.
template <class XV>
YS_HD void spmv_row_sv(const View& v, const double* YS_RESTRICT Ab, int64_t ss, const XV& xv, int n, double y[5]) {
  auto slot = [&](const View&, int s_, int n_) { return Ab[(int64_t)s_ * ss + n_]; };
  const ClothParams& P = v.cp[v.node_cloth[n]];
  const int u = v.node_u[n], w = v.node_v[n];
  double yl0 = 0.0, yl1 = 0.0, yl2 = 0.0;
  for (int s = 0; s < kNumStencil; ++s) {
    const int uu = u + stencil_du(s), vv = w + stencil_dv(s);
    const bool ok = uu >= 0 && uu < P.W && vv >= 0 && vv < P.H;
    const int j = ok ? n + stencil_du(s) + stencil_dv(s) * P.W : n;
    const typename XV::Ptr xp = xv.at(j);
    const double xj0 = xv.get(xp, 0), xj1 = xv.get(xp, 1), xj2 = xv.get(xp, 2);
    const int b = YS_SLOT_LL + 9 * s;
    yl0 = fma(slot(v, b + 0, n), xj0, yl0); yl0 = fma(slot(v, b + 1, n), xj1, yl0); yl0 = fma(slot(v, b + 2, n), xj2, yl0);
    yl1 = fma(slot(v, b + 3, n), xj0, yl1); yl1 = fma(slot(v, b + 4, n), xj1, yl1); yl1 = fma(slot(v, b + 5, n), xj2, yl1);
    yl2 = fma(slot(v, b + 6, n), xj0, yl2); yl2 = fma(slot(v, b + 7, n), xj1, yl2); yl2 = fma(slot(v, b + 8, n), xj2, yl2);
  }
  const typename XV::Ptr xn = xv.at(n);
  const double xu = xv.get(xn, 3), xv_ = xv.get(xn, 4);
  yl0 = fma(slot(v, YS_SLOT_LE_SELF + 0, n), xu, yl0); yl0 = fma(slot(v, YS_SLOT_LE_SELF + 1, n), xv_, yl0);
  yl1 = fma(slot(v, YS_SLOT_LE_SELF + 2, n), xu, yl1); yl1 = fma(slot(v, YS_SLOT_LE_SELF + 3, n), xv_, yl1);
  yl2 = fma(slot(v, YS_SLOT_LE_SELF + 4, n), xu, yl2); yl2 = fma(slot(v, YS_SLOT_LE_SELF + 5, n), xv_, yl2);
  const double xl0 = xv.get(xn, 0), xl1 = xv.get(xn, 1), xl2 = xv.get(xn, 2);
  double ye[2];
  for (int k = 0; k < 2; ++k) {
    double e = slot(v, YS_SLOT_EL_SELF + 3 * k + 0, n) * xl0;
    e = fma(slot(v, YS_SLOT_EL_SELF + 3 * k + 1, n), xl1, e);
    e = fma(slot(v, YS_SLOT_EL_SELF + 3 * k + 2, n), xl2, e);
    ye[k] = fma(slot(v, YS_SLOT_EE_SELF + k, n), k ? xv_ : xu, e);
  }
  for (int m = 0; m < 4; ++m) {
    const int du = m == 0 ? -1 : m == 1 ? 1 : 0, dv = m == 2 ? -1 : m == 3 ? 1 : 0;
    const int k = m < 2 ? 0 : 1;
    const int uu = u + du, vv = w + dv;
    const bool ok = uu >= 0 && uu < P.W && vv >= 0 && vv < P.H;
    const int j = ok ? n + du + dv * P.W : n;
    const typename XV::Ptr xp = xv.at(j);
    const double xe = xv.get(xp, 3 + k);
    yl0 = fma(slot(v, YS_SLOT_LE_NBR + 3 * m + 0, n), xe, yl0);
    yl1 = fma(slot(v, YS_SLOT_LE_NBR + 3 * m + 1, n), xe, yl1);
    yl2 = fma(slot(v, YS_SLOT_LE_NBR + 3 * m + 2, n), xe, yl2);
    ye[k] = fma(slot(v, YS_SLOT_EL_NBR + 3 * m + 0, n), xv.get(xp, 0), ye[k]);
    ye[k] = fma(slot(v, YS_SLOT_EL_NBR + 3 * m + 1, n), xv.get(xp, 1), ye[k]);
    ye[k] = fma(slot(v, YS_SLOT_EL_NBR + 3 * m + 2, n), xv.get(xp, 2), ye[k]);
    ye[k] = fma(slot(v, YS_SLOT_EE_NBR + m, n), xe, ye[k]);
  }
  y[0] = yl0;
  y[1] = yl1;
  y[2] = yl2;
  y[3] = ye[0];
  y[4] = ye[1];
}

YS_HD void spmv_row_s(const View& v, const double* YS_RESTRICT Ab, int64_t ss, const double* YS_RESTRICT x, int n,
                      double y[5]) {
  spmv_row_sv(v, Ab, ss, GlobalVec{x, v.ntot}, n, y);
}

YS_HD void spmv_row(const View& v, const double* YS_RESTRICT x, int n, double y[5]) {
  spmv_row_s(v, v.A, v.ntot, x, n, y);
}

// y = A^T x for row block n: every coefficient that row block i stores for
// column block n (i = n - offset of its slot) is read from row i, transposed.
template <class XV>
YS_HD void spmv_row_tv(const View& v, const XV& xv, int n, double y[5]) {
  const ClothParams& P = v.cp[v.node_cloth[n]];
  const int u = v.node_u[n], w = v.node_v[n];
  double yl[3] = {0.0, 0.0, 0.0}, ye[2] = {0.0, 0.0};
  for (int s = 0; s < kNumStencil; ++s) {
    const int du = stencil_du(s), dv = stencil_dv(s);
    const int uu = u - du, vv = w - dv;  // the row that refers to n through slot s
    if (uu < 0 || uu >= P.W || vv < 0 || vv >= P.H) continue;
    const int i = n - du - dv * P.W;
    const typename XV::Ptr xp = xv.at(i);
    const double x0 = xv.get(xp, 0), x1 = xv.get(xp, 1), x2 = xv.get(xp, 2);
    const int b = YS_SLOT_LL + 9 * s;
    for (int c = 0; c < 3; ++c) {
      yl[c] = fma(slot(v, b + c, i), x0, yl[c]);
      yl[c] = fma(slot(v, b + 3 + c, i), x1, yl[c]);
      yl[c] = fma(slot(v, b + 6 + c, i), x2, yl[c]);
    }
  }
  {  // the node's own Eulerian couplings
    const typename XV::Ptr xp = xv.at(n);
    const double x0 = xv.get(xp, 0), x1 = xv.get(xp, 1), x2 = xv.get(xp, 2);
    for (int k = 0; k < 2; ++k) {
      const double xe = xv.get(xp, 3 + k);
      ye[k] = fma(slot(v, YS_SLOT_LE_SELF + 0 + k, n), x0, ye[k]);
      ye[k] = fma(slot(v, YS_SLOT_LE_SELF + 2 + k, n), x1, ye[k]);
      ye[k] = fma(slot(v, YS_SLOT_LE_SELF + 4 + k, n), x2, ye[k]);
      ye[k] = fma(slot(v, YS_SLOT_EE_SELF + k, n), xe, ye[k]);
      for (int c = 0; c < 3; ++c) yl[c] = fma(slot(v, YS_SLOT_EL_SELF + 3 * k + c, n), xe, yl[c]);
    }
  }
  for (int m = 0; m < 4; ++m) {  // yarn neighbour i = n - offset(m) refers to n through m
    const int du = m == 0 ? -1 : m == 1 ? 1 : 0, dv = m == 2 ? -1 : m == 3 ? 1 : 0;
    const int k = m < 2 ? 0 : 1;
    const int uu = u - du, vv = w - dv;
    if (uu < 0 || uu >= P.W || vv < 0 || vv >= P.H) continue;
    const int i = n - du - dv * P.W;
    const typename XV::Ptr xp = xv.at(i);
    const double xe = xv.get(xp, 3 + k);
    ye[k] = fma(slot(v, YS_SLOT_LE_NBR + 3 * m + 0, i), xv.get(xp, 0), ye[k]);
    ye[k] = fma(slot(v, YS_SLOT_LE_NBR + 3 * m + 1, i), xv.get(xp, 1), ye[k]);
    ye[k] = fma(slot(v, YS_SLOT_LE_NBR + 3 * m + 2, i), xv.get(xp, 2), ye[k]);
    ye[k] = fma(slot(v, YS_SLOT_EE_NBR + m, i), xe, ye[k]);
    for (int c = 0; c < 3; ++c) yl[c] = fma(slot(v, YS_SLOT_EL_NBR + 3 * m + c, i), xe, yl[c]);
  }
  y[0] = yl[0];
  y[1] = yl[1];
  y[2] = yl[2];
  y[3] = ye[0];
  y[4] = ye[1];
}

YS_HD void spmv_row_t(const View& v, const double* YS_RESTRICT x, int n, double y[5]) {
  spmv_row_tv(v, GlobalVec{x, v.ntot}, n, y);
}

// Right-hand side of the tangent solve of row block n for tangent k:
// A dq = db - dA q (q the step's solution; dA, db the tangents of A, b).
YS_HD void tangent_rhs_row(const View& v, const double* YS_RESTRICT q, int n, int k, double r[5]) {
  const int64_t nt = v.ntot;
  double y[5];
  spmv_row_s(v, v.dA + k * nt, (int64_t)v.K * nt, q, n, y);
  for (int c = 0; c < 5; ++c) r[c] = v.dB[((int64_t)c * v.K + k) * nt + n] - (v.trunc ? 0.0 : y[c]);
}

// Cloth::update (src/Cloth.cpp:111-148) for node n with the solved velocity.
YS_HD void update_node(const View& v, const double* YS_RESTRICT xs, int n) {
  const int nt = v.ntot;
  const uint8_t fl = v.flags[n];
  const double h = v.h;
  for (int i = 0; i < 3; ++i) {
    const double vel = xs[i * nt + n];
    st(v.V, i, nt, n) = vel;
    const double x = ld(v.X, i, nt, n) + vel * h;
    st(v.X, i, nt, n) = x;
    if (!(fl & YS_FIXED)) st(v.XF, i, nt, n) = x;
  }
  if (fl & YS_INTERIOR) {
    for (int k = 0; k < 2; ++k) {
      const double e = xs[(3 + k) * nt + n];
      st(v.UVD, k, nt, n) = e;
      st(v.UV, k, nt, n) = ld(v.UV, k, nt, n) + e * h;
      st(v.UVB, k, nt, n) = ld(v.UVB, k, nt, n) + ld(v.SLIDE, k, nt, n) * e * h;
    }
  }
}

// update_node with tangents: xs / dxs hold the solution and its tangents
// ([5][K][ntot]); the state arrays and their tangent arrays are updated
// together (the slide indicator's value is the step's, its tangents dSLIDE).
template <int K>
YS_HD void update_node_dual(const View& v, const double* YS_RESTRICT xs, const double* YS_RESTRICT dxs, double* dX,
                            double* dV, double* dUV, double* dUVD, double* dUVB, int n) {
  typedef Dual<K> D;
  const int nt = v.ntot;
  const uint8_t fl = v.flags[n];
  const double h = v.h;
  for (int i = 0; i < 3; ++i) {
    const D vel = ldT<D>(xs, dxs, i, nt, n);
    stT(v.V, dV, i, nt, n, vel);
    const D x = ldT<D>(v.X, dX, i, nt, n) + vel * h;
    stT(v.X, dX, i, nt, n, x);
    if (!(fl & YS_FIXED)) st(v.XF, i, nt, n) = x.v;
  }
  if (fl & YS_INTERIOR) {
    for (int k = 0; k < 2; ++k) {
      const D e = ldT<D>(xs, dxs, 3 + k, nt, n);
      stT(v.UVD, dUVD, k, nt, n, e);
      stT(v.UV, dUV, k, nt, n, ldT<D>(v.UV, dUV, k, nt, n) + e * h);
      stT(v.UVB, dUVB, k, nt, n,
          ldT<D>(v.UVB, dUVB, k, nt, n) + ldT<D>(v.SLIDE, v.dSLIDE, k, nt, n) * e * h);
    }
  }
}

}  // namespace ys
