// ys_kernels.cu -- CUDA kernels of one implicit step of a batch of cloths.
//
// Assembly: one thread per element writes that element's record (forces and
// Jacobian blocks), then four threads per node gather the records touching its
// row block in a fixed order, so every row is accumulated deterministically
// without atomics.
// Solve: per-cloth Jacobi-PCG (Eigen's ConjugateGradient algorithm, as used by
// src/Solvers.cpp:3-31) on the structured stencil matrix; thread blocks never
// straddle cloths, so each cloth's dot products are a fixed-order sum of its
// blocks' partials, recomputed redundantly by every block that needs them.
#include <cfloat>

#include "ys_pcg.cuh"

namespace ys {

static inline int nblocks(int n) { return (n + kBlock - 1) / kBlock; }

__device__ __forceinline__ void geom_item(const View& v, const int* nodes, int count, int t) {
  if (t >= count) return;
  const int n = nodes[t];
  node_normal(v, n, v.cp[v.node_cloth[n]].W);
}
__global__ void k_geom(View v, const int* __restrict__ nodes, int count) {
  chained();
  geom_item(v, nodes, count, blockIdx.x * blockDim.x + threadIdx.x);
}

// The record producers: one thread per element, nothing shared between
// threads, so any block size gives the same bits; the block size is a schedule
// choice (up to kMaxProducerBlock threads; the edges are compiled for kBlock,
// 128 registers a thread).

// one thread per (yarn direction, node): the edge starting at that node
__device__ __forceinline__ void edge_item(const View& v, const Records& R, int64_t t) {
  if (t >= 2LL * v.ntot) return;
  const int k = t >= v.ntot ? 1 : 0;
  const int n0 = (int)(t - (int64_t)k * v.ntot);
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  if (k == 0 ? v.node_u[n0] >= P.W - 1 : v.node_v[n0] >= P.H - 1) return;
  // each field goes to memory as soon as it is known, so none is held
  edge_terms<double>(v, n0, n0 + (k == 0 ? 1 : P.W), k,
                     [&](int f, double x) { stT(R.edge, R.dedge, 2 * f + k, v.ntot, n0, x); });
}
__global__ void __launch_bounds__(kBlock) k_edge_rec(View v, Records R) {
  chained();
  edge_item(v, R, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// one thread per (yarn direction, middle node) of a bend segment
__global__ void __launch_bounds__(kMaxProducerBlock) k_bend_rec(View v, Records R) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2LL * v.ntot) return;
  const int k = t >= v.ntot ? 1 : 0;
  const int n0 = (int)(t - (int64_t)k * v.ntot);
  const ClothParams& P = v.cp[v.node_cloth[n0]];
  const int pos = k == 0 ? v.node_u[n0] : v.node_v[n0], len = k == 0 ? P.W : P.H;
  if (pos < 1 || pos > len - 2) return;
  const int step = k == 0 ? 1 : P.W;
  const int line = k == 0 ? P.warp_line_off + v.node_v[n0] : P.weft_line_off + v.node_u[n0];
  bend_element<double>(v, R.bend, R.dbend, n0 - step, n0, n0 + step, k, line);
}

// one thread per grid cell (top-left node): its two faces
__device__ __forceinline__ void face_item(const View& v, const Records& R, int n) {
  if (n >= v.ntot) return;
  const ClothParams& P = v.cp[v.node_cloth[n]];
  if (v.node_u[n] >= P.W - 1 || v.node_v[n] >= P.H - 1) return;
  cell_faces<double>(v, R.face, R.dface, n);
}
__global__ void __launch_bounds__(kMaxProducerBlock) k_face_rec(View v, Records R) {
  chained();
  face_item(v, R, blockIdx.x * blockDim.x + threadIdx.x);
}

// What depends on the state alone in one launch, for batches that leave SMs idle
// (Blocks::by_rows) launch by launch: normals, edges, faces, the cloths' status
// cleared. Each of the three is 8 to 20 us of one thread's latency on a small
// cloth. Blocks [0, ng) take the normals, the next ne the edges, the rest faces.
__global__ void __launch_bounds__(kBlock) k_state_rec(View v, Records R, const int* __restrict__ nodes, int count,
                                                      PcgCloth* pc, int ng, int ne) {
  chained();
  const int blk = blockIdx.x;
  if (blk == 0)
    for (int c = threadIdx.x; c < v.ncloth; c += kBlock) pc[c].status = 0;
  if (blk < ng) geom_item(v, nodes, count, blk * kBlock + threadIdx.x);
  else if (blk < ng + ne) edge_item(v, R, (int64_t)(blk - ng) * kBlock + threadIdx.x);
  else face_item(v, R, (blk - ng - ne) * kBlock + threadIdx.x);
}

// one thread per (segment type, crossing)
__global__ void __launch_bounds__(kMaxProducerBlock) k_shear_rec(View v, Records R) {
  chained();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 4LL * v.ntot) return;
  const int seg = (int)(t / v.ntot);
  const int n0 = (int)(t - (int64_t)seg * v.ntot);
  if (!(v.flags[n0] & YS_INTERIOR)) return;
  shear_element<double>(v, R.shear, R.dshear, n0, seg);
}

// ------------------------------------------------------------- the gathers
// A block takes 32 consecutive nodes, warp m their part m (ys_items.cuh), so
// a warp's branches are uniform and its loads whole 256-byte runs; the parts
// meet in shared memory in the order the host code adds them.
constexpr int kNodesPerBlock = 32;

// crossing pass: compression, slide indicator and friction. FP64-latency bound
// (an exp and three tanh behind the sums): the two yarns' frictions run in
// two warps.
__global__ void __launch_bounds__(4 * kNodesPerBlock) k_cross(View v, Records R) {
  chained();
  __shared__ double sc[3][4][kNodesPerBlock], sk[6][4][kNodesPerBlock];
  const int m = threadIdx.x >> 5, i = threadIdx.x & 31;
  const int node = blockIdx.x * kNodesPerBlock + i;
  const bool valid = node < v.ntot;
  const int n = valid ? node : v.ntot - 1;
  const NodeAt N(v, n);
  if (valid && N.in) {
    CrossPart<double> c;
    cross_part(v, R, N, m, c);
    for (int r = 0; r < 3; ++r) { sc[r][m][i] = c.CL[r]; sk[r][m][i] = c.CLE[r]; }
    sk[3][m][i] = c.FE;
    sk[4][m][i] = c.KEE;
    sk[5][m][i] = c.DEE;
  }
  __syncthreads();
  if (m >= 2 || !valid || !N.in) return;
  double CL[3], s[6];
  for (int r = 0; r < 3; ++r) CL[r] = (sc[r][0][i] + sc[r][1][i]) + (sc[r][2][i] + sc[r][3][i]);
  const int k = m;
  for (int r = 0; r < 6; ++r) s[r] = sk[r][2 * k][i] + sk[r][2 * k + 1][i];
  const double comp = crossing_comp(v, n, CL);
  if (k == 0) st(v.COMP, 0, v.ntot, n) = comp;
  double aEE, bE;
  friction_node(v, n, k, comp, s[3], s[4], s[5], s, aEE, bE);
  slot(v, YS_SLOT_EE_SELF + k, n) = aEE;
  st(v.B, 3 + k, v.ntot, n) = bE;
}

// row pass: the 159 slots, b and the Jacobi diagonal of every row block, each
// written once. Latency bound on the record loads: four warps a node hide
// what one thread a node could not. With k_cross, 0.70 ms on 255,292 nodes for
// the 0.97 ms of a gather and a finalize that took one thread a node each and
// passed 81 slots through memory; 34 us for 99 on one 50 x 50 cloth.
__global__ void __launch_bounds__(4 * kNodesPerBlock) k_rows(View v, Records R, Solver so) {
  chained();
  __shared__ double sx[12][4][kNodesPerBlock], se[8][4][kNodesPerBlock], sd[2][9][4][kNodesPerBlock];
  const int m = threadIdx.x >> 5, i = threadIdx.x & 31;
  const int node = blockIdx.x * kNodesPerBlock + i;
  const bool valid = node < v.ntot;
  const int n = valid ? node : v.ntot - 1;
  const NodeAt N(v, n);
  bool fin = true;
  if (valid) {
    RowPart<double> o;
    row_part(v, R, N, m, o, fin, [&](bool mine, int j, double x) { sd[mine ? 0 : 1][j][m][i] = x; });
    for (int j = 0; j < 9; ++j) sx[j][m][i] = o.LL[j];
    for (int r = 0; r < 3; ++r) { sx[9 + r][m][i] = o.B[r]; se[r][m][i] = o.LE[r]; se[3 + r][m][i] = o.EL[r]; }
    se[6][m][i] = o.EE;
    se[7][m][i] = o.Be;
  }
  __syncthreads();
  if (!valid) return;
  const int from = diag_from(m), ds = YS_SLOT_LL + 9 * diag_slot(m);
  for (int j = 0; j < 9; ++j) {
    const double x = sd[0][j][m][i] + sd[1][j][from][i];
    fin = fin && finite_(x);
    slot(v, ds + j, n) = x;
  }
  if (m < 3) {
    double s[4];
    for (int c = 0; c < 4; ++c) {
      const int j = c < 3 ? 3 * m + c : 9 + m;
      s[c] = (sx[j][0][i] + sx[j][1][i]) + (sx[j][2][i] + sx[j][3][i]);
    }
    row_self_x<double>(v, n, m, s, s[3], so.dinv, fin);
  }
  if (m >= 2) {
    const int k = m - 2;
    double s[8];
    for (int c = 0; c < 8; ++c) s[c] = se[c][2 * k][i] + se[c][2 * k + 1][i];
    row_self_e<double>(v, n, k, N.in, s, s + 3, s[6], s[7], so.dinv, fin);
  }
  if (!fin) atomicOr(&so.pc[v.node_cloth[n]].status, 1);
}

// ----------------------------------------------------------------- solve
// sum over the block in thread 0: a tree per warp, then the warps
__device__ __forceinline__ double block_sum(double val, double* sh) {
  for (int o = 16; o > 0; o >>= 1) val += __shfl_down_sync(0xffffffffu, val, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[wid] = val;
  __syncthreads();
  static_assert(kBlock == 128, "four warps");
  return threadIdx.x == 0 ? four_sum(sh[0], sh[1], sh[2], sh[3]) : 0.0;
}

// In a batch that leaves SMs idle (by_rows) a thread's vectors are loaded
// together, before the cloth sum: the loads of one component cannot pass the
// stores of the one before. In one that fills them the registers this takes
// cost more warps than it hides: k_pcg_axpy 28 us for 23 on 255,292 nodes.
__device__ __forceinline__ void load5(const double* p, int64_t nt, int n, bool own, double (&x)[5]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) x[k] = own ? p[k * nt + n] : 0.0;
}

// x = 0, r = b, p = z = Dinv r; partials |r|^2 (row 1, and |b|^2)
// and r.z (row 2)
__global__ void __launch_bounds__(kBlock) k_pcg_setup(View v, Blocks b, Solver so) {
  chained();
  __shared__ double sh[kBlock / 32];
  const int blk = blockIdx.x;
  const int n = b.blk_node0[blk] + threadIdx.x;
  const int nt = v.ntot;
  double rr = 0.0, rz = 0.0;
  if (threadIdx.x < b.blk_count[blk]) {
    for (int k = 0; k < 5; ++k) {
      const double r = ld(v.B, k, nt, n);
      st(so.x, k, nt, n) = 0.0;
      st(so.r, k, nt, n) = r;
      st(so.p, k, nt, n) = pcg_norms(r, ld(so.dinv, k, nt, n), rr, rz);
    }
  }
  double s1 = block_sum(rr, sh);
  if (threadIdx.x == 0) so.part[1 * b.nblk + blk] = s1;
  double s2 = block_sum(rz, sh);
  if (threadIdx.x == 0) so.part[2 * b.nblk + blk] = s2;
}

// one warp per cloth
__global__ void k_pcg_start(Blocks b, Solver so, int ncloth) {
  chained();
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= ncloth) return;
  PcgCloth& pc = so.pc[c];
  const double rr = cloth_sum(b, so.part, 1, c), bb = rr;  // r = b
  const double rz = cloth_sum(b, so.part, 2, c);
  if (threadIdx.x & 31) return;
  pc.bb = bb;
  const double thr = pcg_threshold(so.tol, bb);
  pc.thr = thr;
  pc.rr = rr;
  pc.rz[0] = rz;
  pc.iters = 0;
  pc.active = (pc.status == 0 && bb != 0.0 && rr >= thr) ? 1 : 0;
}

// q = A p and partial p.q (row 0), a thread per node
template <bool TRANS>
__global__ void __launch_bounds__(kBlock) k_pcg_spmv(View v, Blocks b, Solver so) {
  __shared__ double sh[kBlock / 32];
  const int blk = blockIdx.x;
  const int c = b.blk_cloth[blk];
  if (!so.pc[c].active) return;
  const int n = b.blk_node0[blk] + threadIdx.x;
  const int nt = v.ntot;
  double pq = 0.0;
  if (threadIdx.x < b.blk_count[blk]) {
    double y[5];
    if (TRANS) spmv_row_t(v, so.p, n, y);
    else spmv_row(v, so.p, n, y);
    for (int k = 0; k < 5; ++k) {
      st(so.q, k, nt, n) = y[k];
      pq = fma(ld(so.p, k, nt, n), y[k], pq);
    }
  }
  const double s = block_sum(pq, sh);
  if (threadIdx.x == 0) so.part[0 * b.nblk + blk] = s;
}

// The same for batches that leave SMs idle with a thread per node (b.by_rows):
// a group of 32 nodes a block, a warp per part of their rows, the groups'
// partials of p.q. The light part 3 takes turns over the SM's four FP64 pipes.
// Measured, us for 32 products (events): one 17 x 17 cloth 361 for 468, one
// 100 x 100 384 for 502, four 592 for 674 (316 blocks of 128 nodes), 96 of 17 x
// 17 512 for 514 (288), 64 of 40 x 40 1596 for 1151 (832): three warps read
// each x where one did. Hence the line at two blocks an SM.
template <bool TRANS>
__global__ void __launch_bounds__(4 * kGroup) k_pcg_spmv_rows(View v, Blocks b, Solver so) {
  chained();
  __shared__ double sq[5][kGroup];
  const int blk = blockIdx.x >> 2, first = kGroup * (blockIdx.x & 3);
  if (!so.pc[b.blk_cloth[blk]].active) return;
  const int lane = threadIdx.x & 31, m = ((threadIdx.x >> 5) + blockIdx.x) & 3;
  const bool own = first + lane < b.blk_count[blk];
  const int nt = v.ntot, n = own ? b.blk_node0[blk] + first + lane : b.blk_node0[blk];
  const ClothParams& P = v.cp[v.node_cloth[n]];
  const int W = P.W, H = P.H, u = v.node_u[n], w = v.node_v[n];
  auto has = [&](int du, int dv) { return u + du >= 0 && u + du < W && w + dv >= 0 && w + dv < H; };
  auto row = [&](int du, int dv) { return has(-du, -dv) ? n - du - dv * W : -1; };
  const double* A = v.A;
  const double* x = so.p;
  double q[2] = {0.0, 0.0};
  if (own) {
    row_product<TRANS>(
        m, [&](int j) { return row_coef<TRANS>(A, nt, n, m, j, row); },
        [&](int k, int du, int dv) { return x[(int64_t)k * nt + (has(du, dv) ? n + du + dv * W : n)]; }, q);
    st(so.q, m, nt, n) = q[0];
    if (m == 3) st(so.q, 4, nt, n) = q[1];
  }
  sq[m][lane] = q[0];
  if (m == 3) sq[4][lane] = q[1];
  __syncthreads();
  if (m != 3) return;
  double t = 0.0;
  if (own)
#pragma unroll
    for (int k = 0; k < 5; ++k) t = fma(x[(int64_t)k * nt + n], sq[k][lane], t);
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if (lane == 0) so.part[pq_row(b) + blockIdx.x] = t;
}

// alpha = rz / pq; x += alpha p; r -= alpha q; partials |r|^2 (row 1), r.z (row 2)
__global__ void __launch_bounds__(kBlock) k_pcg_axpy(View v, Blocks b, Solver so, int parity) {
  __shared__ double sh[kBlock / 32];
  __shared__ double alpha_sh;
  const int blk = blockIdx.x;
  const int c = b.blk_cloth[blk];
  if (!so.pc[c].active) return;
  if (threadIdx.x < 32) {
    const double pq = cloth_sum(b, so.part, 0, c);
    if (threadIdx.x == 0) alpha_sh = so.pc[c].rz[parity] / pq;
  }
  __syncthreads();
  const double alpha = alpha_sh;
  const int n = b.blk_node0[blk] + threadIdx.x;
  const int nt = v.ntot;
  double rr = 0.0, rz = 0.0;
  if (threadIdx.x < b.blk_count[blk]) {
    for (int k = 0; k < 5; ++k) {
      double x = ld(so.x, k, nt, n), r = ld(so.r, k, nt, n);
      pcg_advance(alpha, ld(so.p, k, nt, n), ld(so.q, k, nt, n), x, r);
      st(so.x, k, nt, n) = x;
      st(so.r, k, nt, n) = r;
      pcg_norms(r, ld(so.dinv, k, nt, n), rr, rz);
    }
  }
  double s1 = block_sum(rr, sh);
  if (threadIdx.x == 0) so.part[1 * b.nblk + blk] = s1;
  double s2 = block_sum(rz, sh);
  if (threadIdx.x == 0) so.part[2 * b.nblk + blk] = s2;
}

// The same where batches leave SMs idle (by_rows)
__global__ void __launch_bounds__(kBlock) k_pcg_axpy_early(View v, Blocks b, Solver so, int parity) {
  chained();
  __shared__ double sh[kBlock / 32];
  __shared__ double alpha_sh;
  const int blk = blockIdx.x, c = b.blk_cloth[blk], nt = v.ntot;
  if (!so.pc[c].active) return;
  const bool own = threadIdx.x < b.blk_count[blk];
  const int n = b.blk_node0[blk] + threadIdx.x;
  double x[5], r[5], p[5], q[5], dinv[5], dot[2] = {0.0, 0.0};
  load5(so.q, nt, n, own, q);
  load5(so.r, nt, n, own, r);
  load5(so.dinv, nt, n, own, dinv);
  load5(so.p, nt, n, own, p);
  load5(so.x, nt, n, own, x);
  if (threadIdx.x < 32) {
    const double pq = cloth_sum_pq(b, so.part, c);
    if (threadIdx.x == 0) alpha_sh = so.pc[c].rz[parity] / pq;
  }
  __syncthreads();
  const double alpha = alpha_sh;
  if (own)
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      pcg_advance(alpha, p[k], q[k], x[k], r[k]);
      st(so.x, k, nt, n) = x[k];
      st(so.r, k, nt, n) = r[k];
      pcg_norms(r[k], dinv[k], dot[0], dot[1]);
    }
  const double s1 = block_sum(dot[0], sh);
  if (threadIdx.x == 0) so.part[1 * b.nblk + blk] = s1;
  const double s2 = block_sum(dot[1], sh);
  if (threadIdx.x == 0) so.part[2 * b.nblk + blk] = s2;
}

// stop test |r|^2 < thr, else beta = rz_new / rz and p = z + beta p. Every
// block of a cloth reaches the same decision from the same fixed-order sums;
// only the cloth's first block writes the cloth's bookkeeping.
template <bool EARLY>
__global__ void __launch_bounds__(kBlock) k_pcg_dir(View v, Blocks b, Solver so, int parity, int it_local) {
  if (EARLY) chained();
  __shared__ int go_sh;
  const int it = so.it_base ? *so.it_base + it_local : it_local;
  __shared__ double beta_sh;
  const int blk = blockIdx.x;
  const int c = b.blk_cloth[blk];
  PcgCloth& pc = so.pc[c];
  if (!pc.active) return;
  const bool own = threadIdx.x < b.blk_count[blk];
  const int n = b.blk_node0[blk] + threadIdx.x, nt = v.ntot;
  double r[5], dinv[5], p[5];
  auto load = [&] {
    load5(so.r, nt, n, own, r);
    load5(so.dinv, nt, n, own, dinv);
    load5(so.p, nt, n, own, p);
  };
  if (EARLY) load();
  if (threadIdx.x < 32) {
    const double rr = cloth_sum(b, so.part, 1, c);
    const double rzn = cloth_sum(b, so.part, 2, c);
    if (threadIdx.x == 0) {
      const bool lead = blk == b.cloth_blk0[c];
      const bool conv = rr < pc.thr;
      // every active cloth has completed exactly `it` iterations before this one
      const bool cap = !conv && it + 1 >= pc.maxiter;
      go_sh = !(conv || cap);
      beta_sh = rzn * (1.0 / pc.rz[parity]);  // (the persistent solve has the reciprocal early)
      if (lead) {
        pc.rr = rr;
        pc.rz[parity ^ 1] = rzn;
        pc.iters = conv ? it : it + 1;
        if (conv || cap) pc.active = 0;
        if (cap) pc.status |= 4;
      }
    }
  }
  __syncthreads();
  if (!go_sh) return;
  if (!EARLY) load();
  const double beta = beta_sh;
  if (own)
#pragma unroll
    for (int k = 0; k < 5; ++k) st(so.p, k, nt, n) = fma(beta, p[k], dinv[k] * r[k]);
}

__global__ void k_count_active(Solver so, int ncloth) {
  chained();
  __shared__ int cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  int mine = 0;
  for (int c = threadIdx.x; c < ncloth; c += blockDim.x) mine += so.pc[c].active;
  atomicAdd(&cnt, mine);
  __syncthreads();
  if (threadIdx.x == 0) *so.nactive = cnt;
}

// flags a cloth whose solution holds a non-finite value (src/TrainHelper.cpp:41-48)
__global__ void __launch_bounds__(kBlock) k_check_solution(View v, Blocks b, Solver so) {
  chained();
  if (so.hold && *so.hold) return;
  const int blk = blockIdx.x;
  const int c = b.blk_cloth[blk];
  const int n = b.blk_node0[blk] + threadIdx.x;
  bool ok = true;
  if (threadIdx.x < b.blk_count[blk])
    for (int k = 0; k < 5; ++k) ok = ok && isfinite(ld(so.x, k, v.ntot, n));
  if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicOr(&so.pc[c].status, 2);
}

// Cloth::update for every cloth whose step succeeded
__global__ void __launch_bounds__(kBlock) k_update(View v, Blocks b, Solver so) {
  chained();
  if (so.hold && *so.hold) return;
  const int blk = blockIdx.x;
  const int c = b.blk_cloth[blk];
  const int n = b.blk_node0[blk] + threadIdx.x;
  if (threadIdx.x >= b.blk_count[blk]) return;
  if (so.pc[c].status & 3) return;  // SimStep returns false and leaves the cloth as it was
  update_node(v, so.x, n);
}

__global__ void k_learned_verdict(Solver so, int ncloth, const int* err, int caller_cap, int* hold) {
  int redo = *err != 0;
  for (int c = threadIdx.x; c < ncloth; c += blockDim.x) {
    const int st = so.pc[c].status;
    if (!(st & 1) && ((st & 8) || ((st & 4) && !caller_cap))) redo = 1;
  }
  redo = __syncthreads_or(redo);
  if (threadIdx.x == 0) *hold = redo;
}

__global__ void k_spmv_plain(View v, const double* x, double* y) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= v.ntot) return;
  double r[5];
  spmv_row(v, x, n, r);
  for (int k = 0; k < 5; ++k) y[(int64_t)k * v.ntot + n] = r[k];
}

// ----------------------------------------------------------------- launchers
void launch_geom(const View& v, const int* nodes, int n, cudaStream_t s) {
  if (n) chain(k_geom, nblocks(n), kBlock, s, v, nodes, n);
}
static inline unsigned pblocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }
void launch_edge_records(const View& v, const Records& R, cudaStream_t s, int t) {
  t = t < kBlock ? t : kBlock;  // k_edge_rec is compiled for at most kBlock threads
  chain(k_edge_rec, pblocks(2LL * v.ntot, t), t, s, v, R);
}
void launch_bend_records(const View& v, const Records& R, cudaStream_t s, int t) {
  chain(k_bend_rec, pblocks(2LL * v.ntot, t), t, s, v, R);
}
void launch_face_records(const View& v, const Records& R, cudaStream_t s, int t) {
  chain(k_face_rec, pblocks(v.ntot, t), t, s, v, R);
}
void launch_state_records(const View& v, const Records& R, const int* nodes, int n, PcgCloth* pc, cudaStream_t s) {
  const unsigned ng = pblocks(n, kBlock), ne = pblocks(2LL * v.ntot, kBlock), nf = pblocks(v.ntot, kBlock);
  chain(k_state_rec, ng + ne + nf, kBlock, s, v, R, nodes, n, pc, (int)ng, (int)ne);
}
void launch_cross(const View& v, const Records& R, cudaStream_t s) {
  chain(k_cross, pblocks(v.ntot, kNodesPerBlock), 4 * kNodesPerBlock, s, v, R);
}
void launch_shear_records(const View& v, const Records& R, cudaStream_t s, int t) {
  chain(k_shear_rec, pblocks(4LL * v.ntot, t), t, s, v, R);
}
void launch_rows(const View& v, const Records& R, const Solver& so, cudaStream_t s) {
  chain(k_rows, pblocks(v.ntot, kNodesPerBlock), 4 * kNodesPerBlock, s, v, R, so);
}
void launch_pcg_setup(const View& v, const Blocks& b, const Solver& so, cudaStream_t s) {
  chain(k_pcg_setup, b.nblk, kBlock, s, v, b, so);
  chain(k_pcg_start, (v.ncloth + 3) / 4, 128, s, b, so, v.ncloth);
}
void launch_pcg_spmv(const View& v, const Blocks& b, const Solver& so, cudaStream_t s) {
  if (b.by_rows) {
    if (so.trans) chain(k_pcg_spmv_rows<true>, 4 * b.nblk, 4 * kGroup, s, v, b, so);
    else chain(k_pcg_spmv_rows<false>, 4 * b.nblk, 4 * kGroup, s, v, b, so);
  } else {
    if (so.trans) k_pcg_spmv<true><<<b.nblk, kBlock, 0, s>>>(v, b, so);
    else k_pcg_spmv<false><<<b.nblk, kBlock, 0, s>>>(v, b, so);
  }
}
void launch_pcg_axpy(const View& v, const Blocks& b, const Solver& so, int it, cudaStream_t s) {
  if (b.by_rows) chain(k_pcg_axpy_early, b.nblk, kBlock, s, v, b, so, it & 1);
  else k_pcg_axpy<<<b.nblk, kBlock, 0, s>>>(v, b, so, it & 1);
}
void launch_pcg_dir(const View& v, const Blocks& b, const Solver& so, int it, cudaStream_t s) {
  if (b.by_rows) chain(k_pcg_dir<true>, b.nblk, kBlock, s, v, b, so, it & 1, it);
  else k_pcg_dir<false><<<b.nblk, kBlock, 0, s>>>(v, b, so, it & 1, it);
}
void launch_count_active(const View& v, const Solver& so, cudaStream_t s) {
  chain(k_count_active, 1, 256, s, so, v.ncloth);
}
__global__ void k_graph_loop_begin(Solver so) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *so.it_base = 0;
}
__global__ void k_graph_loop_tail(Solver so, int ncloth, int m, int cap, cudaGraphConditionalHandle h) {
  __shared__ int cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  int mine = 0;
  for (int c = threadIdx.x; c < ncloth; c += blockDim.x) mine += so.pc[c].active;
  atomicAdd(&cnt, mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    *so.nactive = cnt;
    const int done = *so.it_base + m;
    *so.it_base = done;
    // the loop ends when no cloth iterates or at the iteration cap, whichever first
    cudaGraphSetConditional(h, (cnt > 0 && done < cap) ? 1u : 0u);
  }
}
void launch_graph_loop_begin(const Solver& so, cudaStream_t s) { k_graph_loop_begin<<<1, 32, 0, s>>>(so); }
void launch_graph_loop_tail(const Solver& so, int ncloth, int m, int cap, cudaGraphConditionalHandle h,
                            cudaStream_t s) {
  k_graph_loop_tail<<<1, 256, 0, s>>>(so, ncloth, m, cap, h);
}
void launch_check_solution(const View& v, const Blocks& b, const Solver& so, cudaStream_t s) {
  chain(k_check_solution, b.nblk, kBlock, s, v, b, so);
}
void launch_update(const View& v, const Blocks& b, const Solver& so, cudaStream_t s) {
  chain(k_check_solution, b.nblk, kBlock, s, v, b, so);
  chain(k_update, b.nblk, kBlock, s, v, b, so);
}
void launch_learned_verdict(const Solver& so, int ncloth, const int* err, int caller_cap, int* hold,
                            cudaStream_t s) {
  k_learned_verdict<<<1, 256, 0, s>>>(so, ncloth, err, caller_cap, hold);
}
void launch_spmv(const View& v, const double* x, double* y, cudaStream_t s) {
  k_spmv_plain<<<nblocks(v.ntot), kBlock, 0, s>>>(v, x, y);
}

}  // namespace ys
