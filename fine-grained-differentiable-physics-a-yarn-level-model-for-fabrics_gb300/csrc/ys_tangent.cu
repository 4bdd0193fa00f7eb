// ys_tangent.cu -- forward-mode sensitivity kernels of one step: the
// right-hand sides of the tangent solves and the update of state tangents.
//
// A direction's tangent solve is A dq = db - dA q (q the step's solution), or
// db alone in the reference mode: only the tangent of the residual b - A q at
// fixed q is needed, never those of the 159 coefficients. One thread per
// (direction, element) evaluates the element code (ys_physics.cuh) over
// Dual<1> and folds each field it yields with q at once; what reaches memory
// is the element's residual (8 to 12 numbers) and, for friction, the tangents
// of the gathered forces. Bound by FP64 latency on small cloths (the shear
// terms' chains at 250 registers). Two 17 x 17 copies with four directions:
// 0.96 ms a step (5.59 with the five solves one after another, as when these
// kernels came), for 7.26 ms with records and rows over Dual<4>, which spilled 2
// to 8 KB a thread and wrote 159 tangents a node and direction; 4.5 KB of
// buffers a node for 21.
#include "ys_items.cuh"
#include "ys_kernels.cuh"

namespace ys {

namespace {

constexpr int K = kTangents;
typedef Dual<1> D1;

// residual fields per element: edges r(n0) 4, r(n1) 4, crimp force 3 and its
// Eulerian derivative 3, F_E 2, dF_E/dE 2, dF_E/dE' 2; bend segments r(n2) 4,
// r(n0) 4, r(n1) 4, crimp forces 6, dF_E/dE, F_E at n2
constexpr int kTE_r = 0, kTE_cl = 8, kTE_cle = 11, kTE_fe = 14, kTE_kee = 16, kTE_dee = 18, kTE = 20;
constexpr int kTB_r = 0, kTB_cF1 = 12, kTB_cF2 = 15, kTB_E = 18, kTB_F = 19, kTB = 20;
constexpr int kTF = 6;
constexpr int kTS = 6;  // r(n1) 3, r(n3) 3
constexpr int kTC = 2;  // friction's share of the Eulerian rows
static_assert(2 * kTE + 2 * kTB + kTF + 4 * kTS + kTC == kTangentScratch, "tangent scratch");

// the view of direction k alone: its tangent arrays at the direction's offset
// (Dual<1> loads keep the stride of the kTangents directions, lds)
__device__ __forceinline__ View direction(const View& v, int k) {
  View d = v;
  const int64_t o = (int64_t)k * v.ntot;
  d.dX += o; d.dV += o; d.dUV += o; d.dUVD += o; d.dUVB += o;
  d.dNRM += o; d.dCOMP += o; d.dSLIDE += o;
  d.dline_rho += (int64_t)k * v.nlines; d.dline_ks += (int64_t)k * v.nlines; d.dline_kb += (int64_t)k * v.nlines;
  d.dS += (int64_t)k * v.ncloth;
  d.dmu += (int64_t)k * v.ncloth;
  return d;
}

// direction k's scratch
struct Scratch {
  double *edge, *bend, *face, *shear, *cross;
  __device__ __forceinline__ Scratch(double* base, int k, int64_t nt) {
    edge = base + (int64_t)k * kTangentScratch * nt;
    bend = edge + 2 * kTE * nt;
    face = bend + 2 * kTB * nt;
    shear = face + kTF * nt;
    cross = shear + 4 * kTS * nt;
  }
};

}  // namespace

// Tangents of the normals: the stencil's scatter matrix S changes by dS
__global__ void __launch_bounds__(64) k_tan_geom(View v, const int* __restrict__ nodes, int count) {
  chained();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int n = nodes[t], nt = v.ntot, W = v.cp[v.node_cloth[n]].W;
  const int ids[5] = {n, n - 1, n + 1, n - W, n + W};
  double p[5][3], mean[3] = {0, 0, 0}, S[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, nn[3];
  for (int m = 0; m < 5; ++m)
    for (int i = 0; i < 3; ++i) { p[m][i] = ld(v.X, i, nt, ids[m]); mean[i] += p[m][i]; }
  for (int m = 0; m < 5; ++m)
    for (int i = 0; i < 3; ++i) p[m][i] -= mean[i] / 5.0;
  for (int m = 0; m < 5; ++m)
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) S[i][j] += p[m][i] * p[m][j];
  for (int i = 0; i < 3; ++i) nn[i] = ld(v.NRM, i, nt, n);
  const NormalResponse N(S, nn);
  for (int k = 0; k < K; ++k) {
    double g[3] = {0, 0, 0}, dn[3];  // dS n (the mean's share sums to 0)
    for (int m = 0; m < 5; ++m) {
      double x[3], rn = 0.0, xn = 0.0;
      for (int i = 0; i < 3; ++i) {
        x[i] = v.dX[((int64_t)i * K + k) * nt + ids[m]];
        rn += p[m][i] * nn[i];
        xn += x[i] * nn[i];
      }
      for (int i = 0; i < 3; ++i) g[i] += x[i] * rn + p[m][i] * xn;
    }
    N.respond(g, dn);
    for (int i = 0; i < 3; ++i) v.dNRM[((int64_t)i * K + k) * nt + n] = dn[i];
  }
}

// q: the solution, null in the reference mode (no dA q)
__global__ void __launch_bounds__(64) k_tan_edge(View v, const double* q, double* scratch) {
  chained();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= 2 * nt) return;
  const int k = t >= nt ? 1 : 0, n0 = t - k * nt;
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  if (k == 0 ? v.node_u[n0] >= P.W - 1 : v.node_v[n0] >= P.H - 1) return;
  const int nd[2] = {n0, n0 + (k == 0 ? 1 : P.W)};
  double x[2][4], r[8] = {0, 0, 0, 0, 0, 0, 0, 0}, u[3];
  for (int a = 0; a < 2; ++a)
    for (int i = 0; i < 4; ++i) x[a][i] = q ? q[(int64_t)(i < 3 ? i : 3 + k) * nt + nd[a]] : 0.0;
  for (int i = 0; i < 3; ++i) u[i] = x[1][i] - x[0][i];
  double* out = Scratch(scratch, blockIdx.y, nt).edge + (int64_t)k * nt + n0;
  auto put = [&](int f, double y) { out[(int64_t)f * 2 * nt] = y; };
  D1 lP, cl, cle, d[3];
  edge_terms(edge_load<D1>(direction(v, blockIdx.y), nd[0], nd[1], k), P, k, v.h, v.trunc != 0,
             [&](int f, const D1& y) {
               const double t = y.d[0];
               if (f < kE_lP) {
                 const int a = f >> 1, c = f & 1;
                 for (int i = 0; i < 3; ++i) r[4 * a + i] -= t * x[c][i];
               } else if (f == kE_lP) {
                 lP = y;
               } else if (f < kE_le) {
                 const int i = f - kE_d;
                 d[i] = y;
                 put(kTE_cl + i, (cl * y).d[0]);
                 put(kTE_cle + i, (cle * y).d[0]);
                 if (i == 2) {
                   const D1 du = u[0] * d[0] + u[1] * d[1] + u[2] * d[2];
                   for (int j = 0; j < 3; ++j) {  // stretch: lP (I - d d^T) between the ends
                     const double g = (lP * (u[j] - d[j] * du)).d[0];
                     r[j] += g;
                     r[4 + j] -= g;
                   }
                 }
               } else if (f < kE_el) {
                 const int p = (f - kE_le) / 3;
                 r[4 * (p >> 1) + f - kE_le - 3 * p] -= t * x[p & 1][3];
               } else if (f < kE_ee) {
                 const int p = (f - kE_el) / 3;
                 r[4 * (p >> 1) + 3] -= t * x[p & 1][f - kE_el - 3 * p];
               } else if (f < kE_b) {
                 const int p = f - kE_ee;
                 r[4 * (p >> 1) + 3] -= t * x[p & 1][3];
               } else if (f < kE_fe) {
                 r[f - kE_b] += t;
               } else if (f == kE_cl) {
                 cl = y;
               } else if (f == kE_cle) {
                 cle = y;
               } else {
                 put(kTE_fe + f - kE_fe, t);  // fe, kee, dee follow each other in both layouts
               }
             });
  for (int i = 0; i < 8; ++i) put(kTE_r + i, r[i]);
}

__global__ void __launch_bounds__(64) k_tan_bend(View v, const double* q, double* scratch) {
  chained();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= 2 * nt) return;
  const int k = t >= nt ? 1 : 0, n0 = t - k * nt;
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  const int pos = k == 0 ? v.node_u[n0] : v.node_v[n0], len = k == 0 ? P.W : P.H;
  if (pos < 1 || pos > len - 2) return;
  const int step = k == 0 ? 1 : P.W, n1 = n0 + step, n2 = n0 - step;
  const int line = k == 0 ? P.warp_line_off + v.node_v[n0] : P.weft_line_off + v.node_u[n0];
  const bool in0 = (v.flags[n0] & YS_INTERIOR) != 0, in1 = (v.flags[n1] & YS_INTERIOR) != 0,
             in2 = (v.flags[n2] & YS_INTERIOR) != 0;
  const double h = v.h, mh2 = -(v.h * v.h);
  double q0[3], q1[3], q2[3], u[3], w[3];
  auto Q = [&](int c, int n) { return q ? q[(int64_t)c * nt + n] : 0.0; };
  for (int i = 0; i < 3; ++i) {
    q0[i] = Q(i, n0);
    q1[i] = Q(i, n1);
    q2[i] = Q(i, n2);
    u[i] = q1[i] - q0[i];
    w[i] = q2[i] - q0[i];
  }
  const double e1 = in1 ? Q(3 + k, n1) : 0.0, e2 = in2 ? Q(3 + k, n2) : 0.0;
  // residuals of n1 and n2 that n0's mirrors (m1, m2), and the rest
  double m1[3] = {0, 0, 0}, m2[3] = {0, 0, 0}, x0[3] = {0, 0, 0}, x1[3] = {0, 0, 0}, x2[3] = {0, 0, 0};
  double r0 = 0.0, r1 = 0.0, r2 = 0.0;
  double* out = Scratch(scratch, blockIdx.y, nt).bend + (int64_t)k * nt + n0;
  auto put = [&](int f, double y) { out[(int64_t)f * 2 * nt] = y; };
  D1 idu;
  bend_terms<D1>(direction(v, blockIdx.y), n2, n0, n1, k, line, [&](int f, const D1& y) {
    const double t = y.d[0];
    if (f < kB_L12) {
      const bool one = f < kB_L22;
      const int g = one ? f : f - kB_L22;
      const int i = g < 3 ? 0 : g < 5 ? 1 : 2, j = g < 3 ? g : g < 5 ? g - 2 : 2;
      double* m = one ? m1 : m2;
      const double* x = one ? u : w;
      m[i] -= t * x[j];
      if (i != j) m[j] -= t * x[i];
    } else if (f < kB_F1) {
      const int i = (f - kB_L12) / 3, j = f - kB_L12 - 3 * i;
      m2[i] -= t * u[j];
      m1[j] -= t * w[i];
    } else if (f < kB_idu) {
      const bool one = f < kB_F2;
      const int i = f - (one ? kB_F1 : kB_F2);
      (one ? m1 : m2)[i] += h * t;
      // the Eulerian couplings: g = -h^2 F / du
      const double g = mh2 * (idu * y).d[0];
      if (one) {
        x1[i] += g * e1;
        if (in1) r1 += g * q1[i];
      } else {
        x2[i] -= g * e2;
        if (in2) r2 -= g * q2[i];
      }
      if (in0 && in2) { x0[i] += g * e2; r0 += g * q2[i]; }
      if (in0 && in1) { x0[i] -= g * e1; r1 -= g * q0[i]; }
    } else if (f == kB_idu) {
      idu = y;
    } else if (f == kB_E1E1) {
      if (in1) r1 -= mh2 * t * e1;
      if (in2) r2 -= mh2 * t * e2;
      put(kTB_E, t);
    } else if (f == kB_Fu2) {
      if (in1) r1 -= h * t;
      if (in2) r2 += h * t;
      put(kTB_F, t);
    } else if (f != kB_cidu) {
      put(kTB_cF1 + f - kB_cF1, t);  // cF1, cF2
    }
  });
  for (int i = 0; i < 3; ++i) {
    put(kTB_r + i, m2[i] + x2[i]);
    put(kTB_r + 4 + i, x0[i] - (m1[i] + m2[i]));
    put(kTB_r + 8 + i, m1[i] + x1[i]);
  }
  put(kTB_r + 3, r2);
  put(kTB_r + 7, r0);
  put(kTB_r + 11, r1);
}

__global__ void __launch_bounds__(64) k_tan_face(View v, double* scratch) {
  chained();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (n >= 2 * nt) return;
  const int which = n >= nt ? 1 : 0, tl = n - which * nt;
  const ClothParams& P = v.cp[v.node_cloth[tl]];
  if (v.node_u[tl] >= P.W - 1 || v.node_v[tl] >= P.H - 1) return;
  int f[3];
  cell_face(v, tl, which, f);
  D1 f3[3];
  wind_face(direction(v, blockIdx.y), P, f[0], f[1], f[2], f3);
  double* out = Scratch(scratch, blockIdx.y, nt).face;
  for (int i = 0; i < 3; ++i) out[(int64_t)(3 * which + i) * nt + tl] = f3[i].d[0];
}

// Compression and friction at the crossings (k_cross): values from the step's
// records R, tangents from the scratch; writes dCOMP, dSLIDE and the tangent
// of bE - aEE q
__global__ void __launch_bounds__(128) k_tan_cross(View v, Records R, const double* q, double* scratch) {
  chained();
  __shared__ double sc[3][4][32], sk[6][4][32], tc[3][4][32], tk[6][4][32];
  const int m = threadIdx.x >> 5, i = threadIdx.x & 31;
  const int node = blockIdx.x * 32 + i;
  const bool valid = node < v.ntot;
  const int n = valid ? node : v.ntot - 1, nt = v.ntot;
  const NodeAt N(v, n);
  const Scratch S(scratch, blockIdx.y, nt);
  if (valid && N.in) {
    CrossPart<double> c;
    cross_part(v, R, N, m, c);
    double t[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};  // CL 3, CLE 3, FE, KEE, DEE
    const int k = part_k(m), dir = part_dir(m), step = N.step(k), pos = N.pos(k), len = N.len(k);
    const double sgn = k == 0 ? 1.0 : -1.0;
    {  // (an interior crossing has all four edges)
      const int a = dir > 0 ? 0 : 1;
      const double* e = S.edge + (int64_t)k * nt + (dir > 0 ? n : n - step);
      auto E = [&](int f) { return e[(int64_t)f * 2 * nt]; };
      for (int r = 0; r < 3; ++r) {
        t[r] += dir > 0 ? E(kTE_cl + r) : -E(kTE_cl + r);
        t[3 + r] += E(kTE_cle + r);
      }
      t[6] += E(kTE_fe + a);
      t[7] += E(kTE_kee + a);
      t[8] += E(kTE_dee + a);
    }
    const int mid = pos + dir;
    if (mid >= 1 && mid <= len - 2) {
      const int b0 = n + dir * step;
      const double* e = S.bend + (int64_t)k * nt + b0;
      auto Bf = [&](int f) { return e[(int64_t)f * 2 * nt]; };
      const double icu = dir * sgn * crimp_icu(v, b0 - step, b0 + step, k);
      for (int r = 0; r < 3; ++r) {
        const double cF = Bf((dir > 0 ? kTB_cF2 : kTB_cF1) + r);
        t[r] += sgn * cF;
        t[3 + r] += icu * cF;
      }
      t[7] += Bf(kTB_E);
      t[6] += dir * Bf(kTB_F);
    }
    if (dir > 0) {
      const double* e = S.bend + (int64_t)k * nt + n;
      for (int r = 0; r < 3; ++r) t[r] -= sgn * (e[(int64_t)(kTB_cF1 + r) * 2 * nt] + e[(int64_t)(kTB_cF2 + r) * 2 * nt]);
    }
    for (int r = 0; r < 3; ++r) {
      sc[r][m][i] = c.CL[r];
      tc[r][m][i] = t[r];
      sk[r][m][i] = c.CLE[r];
      tk[r][m][i] = t[3 + r];
    }
    sk[3][m][i] = c.FE;
    sk[4][m][i] = c.KEE;
    sk[5][m][i] = c.DEE;
    for (int r = 0; r < 3; ++r) tk[3 + r][m][i] = t[6 + r];
  }
  __syncthreads();
  if (m >= 2 || !valid || !N.in) return;
  const int k = m;
  const View d = direction(v, blockIdx.y);
  D1 CL[3], s[6];
  for (int r = 0; r < 3; ++r) {
    CL[r].v = (sc[r][0][i] + sc[r][1][i]) + (sc[r][2][i] + sc[r][3][i]);
    CL[r].d[0] = (tc[r][0][i] + tc[r][1][i]) + (tc[r][2][i] + tc[r][3][i]);
  }
  for (int r = 0; r < 6; ++r) {
    s[r].v = sk[r][2 * k][i] + sk[r][2 * k + 1][i];
    s[r].d[0] = tk[r][2 * k][i] + tk[r][2 * k + 1][i];
  }
  const D1 comp = crossing_comp(d, n, CL);
  if (k == 0) d.dCOMP[n] = comp.d[0];
  D1 ce = 0.0, slide, aEE, bE;
  for (int r = 0; r < 3; ++r) ce += ldT<D1>(d.NRM, d.dNRM, r, nt, n) * s[r];
  const int c = v.node_cloth[n];
  friction_terms(v.cp[c], v.h, v.trunc != 0, comp, 0.5 * ce, cloth_mu<D1>(d, c),
                 ldT<D1>(d.UV, d.dUV, k, nt, n) - ldT<D1>(d.UVB, d.dUVB, k, nt, n),
                 ldT<D1>(d.UVD, d.dUVD, k, nt, n), s[3], s[4], s[5], slide, aEE, bE);
  d.dSLIDE[(int64_t)k * K * nt + n] = slide.d[0];
  S.cross[(int64_t)k * nt + n] = bE.d[0] - (q ? aEE.d[0] * q[(int64_t)(3 + k) * nt + n] : 0.0);
}

__global__ void __launch_bounds__(64) k_tan_shear(View v, const double* q, double* scratch) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot;
  if (t >= 4LL * nt) return;
  const int seg = (int)(t / nt), n0 = (int)(t - (int64_t)seg * nt);
  if (!(v.flags[n0] & YS_INTERIOR)) return;
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  const int n1 = n0 + shear_du(seg), n3 = n0 + shear_dv(seg) * P.W;
  double u[3], x[3], r1[3] = {0, 0, 0}, r3[3] = {0, 0, 0};
  for (int i = 0; i < 3; ++i) {
    u[i] = q ? q[(int64_t)i * nt + n1] - q[(int64_t)i * nt + n0] : 0.0;
    x[i] = q ? q[(int64_t)i * nt + n3] - q[(int64_t)i * nt + n0] : 0.0;
  }
  shear_terms(shear_load<D1>(direction(v, blockIdx.y), n0, seg), P, v.h, v.trunc != 0, [&](int f, const D1& y) {
    const double t = y.d[0];
    if (f < kS_F3) r1[f] += t;
    else if (f < kS_J11) r3[f - kS_F3] += t;
    else {
      const int g = f - kS_J11, blk = g / 9, r = (g - 9 * blk) / 3, c = g - 9 * blk - 3 * r;  // J11, J13, J31, J33
      (blk < 2 ? r1 : r3)[r] -= t * (blk == 0 || blk == 2 ? u[c] : x[c]);
    }
  });
  double* out = Scratch(scratch, blockIdx.y, nt).shear + (int64_t)seg * nt + n0;
  for (int i = 0; i < 3; ++i) {
    out[(int64_t)i * 4 * nt] = r1[i];
    out[(int64_t)(3 + i) * 4 * nt] = r3[i];
  }
}

// rt[k][c][ntot]: every element's residual at node n, one thread per
// (component, node); dext (or null) [kact][ntot][5]: the external force's
// tangents, which add h dext where the rows add h ext
__global__ void __launch_bounds__(128) k_tan_gather(View v, double* scratch, const double* dext,
                                                    double* rt) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nt = v.ntot, dirn = blockIdx.y;
  if (t >= 5LL * nt) return;
  const int c = (int)(t / nt), n = (int)(t - (int64_t)c * nt);
  const NodeAt N(v, n);
  const Scratch S(scratch, dirn, nt);
  auto E = [&](int f, int k, int a) { return S.edge[(int64_t)f * 2 * nt + (int64_t)k * nt + a]; };
  auto B = [&](int f, int k, int a) { return S.bend[(int64_t)f * 2 * nt + (int64_t)k * nt + a]; };
  double s = 0.0;
  const bool e = c >= 3;
  if (e && !N.in) {
    rt[((int64_t)dirn * 5 + c) * nt + n] = 0.0;
    return;
  }
  const int comp = e ? 3 : c;
  for (int k = e ? c - 3 : 0; k <= (e ? c - 3 : 1); ++k) {
    const int step = N.step(k), pos = N.pos(k), len = N.len(k);
    if (pos < len - 1) s += E(kTE_r + comp, k, n);
    if (pos > 0) s += E(kTE_r + 4 + comp, k, n - step);
    if (pos + 1 >= 1 && pos + 1 <= len - 2) s += B(kTB_r + comp, k, n + step);      // n2 of the next segment
    if (pos >= 1 && pos <= len - 2) s += B(kTB_r + 4 + comp, k, n);                 // its middle
    if (pos - 1 >= 1 && pos - 1 <= len - 2) s += B(kTB_r + 8 + comp, k, n - step);  // n1 of the last
  }
  if (e) {
    s += S.cross[(int64_t)(c - 3) * nt + n];
  } else {
    for (int m = 0; m < 4; ++m) {  // wind on the cells around the node (as row_part)
      const int ci = N.u - 1 + (m & 1), cj = N.w - 1 + (m >> 1);
      if (ci < 0 || ci >= N.W - 1 || cj < 0 || cj >= N.H - 1) continue;
      const int tl = n + (ci - N.u) + (cj - N.w) * N.W;
      const bool right = ci != N.u, below = cj != N.w, even = ((ci + cj) & 1) == 0;
      if (!below || right == even) s += v.h * S.face[(int64_t)c * nt + tl];
      if (below || right != even) s += v.h * S.face[(int64_t)(3 + c) * nt + tl];
    }
    for (int seg = 0; seg < 4; ++seg) {
      const int du = shear_du(seg), dv = shear_dv(seg);
      auto H = [&](int f, int a) { return S.shear[(int64_t)f * 4 * nt + (int64_t)seg * nt + a]; };
      if (N.in) s -= H(c, n) + H(3 + c, n);
      if (N.interior(N.u - du, N.w)) s += H(c, n - du);
      if (N.interior(N.u, N.w - dv)) s += H(3 + c, n - dv * N.W);
    }
    if (v.flags[n] & YS_FIXED) s -= v.h * v.cp[v.node_cloth[n]].kh * v.dX[((int64_t)c * K + dirn) * nt + n];
  }
  if (dext) s += v.h * dext[((int64_t)dirn * nt + n) * 5 + c];
  rt[((int64_t)dirn * 5 + c) * nt + n] = s;
}

// Cloth::update of state and tangents for every cloth whose step succeeded
__global__ void __launch_bounds__(kBlock) k_update_dual(View v, Blocks b, Solver so, const double* dq,
                                                        TangentState ts) {
  chained();
  const int blk = blockIdx.x;
  const int c = b.blk_cloth[blk];
  const int n = b.blk_node0[blk] + threadIdx.x;
  if (threadIdx.x >= b.blk_count[blk]) return;
  if (so.pc[c].status & 3) return;
  update_node_dual<kTangents>(v, so.x, dq, ts.dX, ts.dV, ts.dUV, ts.dUVD, ts.dUVB, n);
}

int launch_tangent_residual(const View& v, const Records& R, const int* interior, int n_interior, const double* q,
                            double* scratch, const double* dext, int kact, double* rt, cudaStream_t s) {
  const int64_t nt = v.ntot;
  const double* x = v.trunc ? nullptr : q;
  auto grid = [](int64_t n, int t, int k) { return dim3((unsigned)((n + t - 1) / t), (unsigned)k); };
  chain(k_tan_geom, grid(n_interior, 64, 1), 64, s, v, interior, n_interior);
  chain(k_tan_edge, grid(2 * nt, 64, K), 64, s, v, x, scratch);
  chain(k_tan_bend, grid(2 * nt, 64, K), 64, s, v, x, scratch);
  chain(k_tan_face, grid(2 * nt, 64, K), 64, s, v, scratch);
  chain(k_tan_cross, grid(nt, 32, K), 128, s, v, R, x, scratch);
  chain(k_tan_shear, grid(4 * nt, 64, K), 64, s, v, x, scratch);
  if (kact > 0) chain(k_tan_gather, grid(5 * nt, 128, kact), 128, s, v, scratch, dext, rt);
  return 7;
}
void launch_update_dual(const View& v, const Blocks& b, const Solver& so, const double* dq, const TangentState& ts,
                        cudaStream_t s) {
  launch_check_solution(v, b, so, s);
  chain(k_update_dual, b.nblk, kBlock, s, v, b, so, dq, ts);
}

}  // namespace ys
