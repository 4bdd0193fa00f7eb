// ys_pcg_cluster.cu -- the persistent per-cloth Jacobi-PCG: one thread-block
// cluster runs one cloth's whole solve (set-up, every iteration, the stop
// test) in a single launch.
//
// A CTA owns `groups` groups of 32 consecutive nodes, a group has four warps:
// warp m < 3 computes row m of the node's x rows, 45 of the row block's 159
// coefficients, warp 3 the two Eulerian rows, 24. An SM issues one warp's
// FP64 instruction over 64 cycles of one of its four pipes, so with a thread
// per node a group's product took 159 x 64 cycles of one pipe while the other
// three waited; split by rows the sums keep their order, so the bits are those
// of a thread per node. Each warp keeps its rows' solution, residual and
// inverse diagonal in registers for the whole solve (and, one group a CTA, its
// coefficients).
//
// The direction sits in each CTA's shared memory for the CTA's own nodes and
// the two cloth rows on either side that their stencils reach. z = D^-1 r is
// what the CTAs exchange: it is published with the |r|^2 and r.z partials, and
// after the sums every CTA forms p = z + beta p on its whole window, the same
// bits for a node in every window it lies in. So an iteration has two cluster
// barriers, after the p.q partials and after the others.
//
// The arithmetic is the batched PCG's (k_pcg_setup, k_pcg_spmv, k_pcg_axpy,
// k_pcg_dir in ys_kernels.cu) term for term, and the dot products are summed
// in its order: the components of a node chained, a warp shuffle tree per 32
// nodes, the four group sums of each 128-node block (four_sum), then the
// cloth's blocks (lanes_sum). So the two schedules give the same bits, and both
// restate Eigen's ConjugateGradient with its diagonal preconditioner
// (src/Solvers.cpp:3-31).
#include <cooperative_groups.h>

#include <cfloat>
#include <cstdint>

#include "ys_pcg.cuh"

namespace cg = cooperative_groups;

namespace ys {

namespace {

constexpr int kMaxGroups = 8;      // groups of a CTA
constexpr int kMaxCluster = 16;    // CTAs of a cluster
constexpr int kMaxBlocks = kMaxCluster * kMaxGroups / 4;  // 128-node blocks of a cloth: one per lane
static_assert(kMaxBlocks <= 32 && kGroup == 32, "one block partial per lane");
static_assert(kMaxCluster * kMaxGroups * kGroup == kClusterMaxNodes, "nodes of a cluster");

// the window of a CTA: the nodes [lo, hi) of the cloth that the stencils of its
// own nodes reach
struct Window {
  int lo, hi;
  __host__ __device__ Window(int first, int nodes, int W, int N) {
    lo = first - 2 * W > 0 ? first - 2 * W : 0;
    hi = first + nodes + 2 * W < N ? first + nodes + 2 * W : N;
    if (first >= N) lo = hi = N;  // a CTA without nodes
  }
  __host__ __device__ int size() const { return hi - lo; }
};

// T: most threads a CTA (128 per group); HOLD: coefficients in registers
template <int T, bool CLUSTER, bool TRANS, bool HOLD>
__global__ void __launch_bounds__(T, T <= 256 ? 2 : 1) k_pcg_cluster(View v, Solver so, ClusterRhs io, const int* __restrict__ cloths, int cap) {
  extern __shared__ double dyn[];
  __shared__ double gp[2][2][kMaxGroups];  // group partials of two dot products, alternating
  __shared__ double out[2], irz;
  const int groups = blockDim.x / (4 * kGroup), own_nodes = groups * kGroup;
  double* zs = dyn;                    // [5][own_nodes] z, read by the other CTAs
  double* rs = dyn + 5 * own_nodes;    // [5][own_nodes] q, then r, for the dot products
  double* sp = dyn + 10 * own_nodes;   // [5][window] direction
  const int csize = CLUSTER ? (int)cg::this_cluster().num_blocks() : 1;
  const int rank = CLUSTER ? (int)cg::this_cluster().block_rank() : 0;
  const int c = cloths[blockIdx.x / csize];
  const int rhs = blockIdx.y;
  PcgCloth& pc = io.pc[(int64_t)rhs * v.ncloth + c];
  const double* __restrict__ b = io.b + rhs * io.b_rhs;
  const ClothParams& P = v.cp[c];
  const int W = P.W, H = P.H, N = W * H, off = P.node_off, nt = v.ntot;
  const int nblk = (N + kBlock - 1) / kBlock;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, grp = wid >> 2;
  const int m = (wid + grp) & 3;  // a group's light warp 3 on another pipe than the next group's
  const int nc = m == 3 ? 2 : 1;
  const int at = grp * kGroup + lane, li = rank * own_nodes + at;
  const bool own = li < N;
  const int n = off + (own ? li : 0);
  const int u = v.node_u[n], w = v.node_v[n];
  const Window win(rank * own_nodes, own_nodes, W, N);
  const int WN = win.size(), pos = own ? li - win.lo : 0;
  const int maxiter = pc.maxiter;
  const bool ok_sys = pc.status == 0;  // read before any CTA of the cluster can write it
  const double* __restrict__ A = v.A;
  auto sync_all = [&] {
    if (CLUSTER) cg::this_cluster().sync();
    else __syncthreads();
  };
  auto has = [&](int du, int dv) { return u + du >= 0 && u + du < W && w + dv >= 0 && w + dv < H; };
  // A^T: the row that refers to this node through (du, dv) lies opposite
  auto row = [&](int du, int dv) { return has(-du, -dv) ? n - du - dv * W : -1; };
  auto coef = [&](int j) { return row_coef<TRANS>(A, nt, n, m, j, row); };
  auto x_at = [&](int k, int du, int dv) { return sp[k * WN + (has(du, dv) ? pos + du + dv * W : pos)]; };
  // the chain over a node's components and the tree over the group's nodes;
  // lane 0 keeps the group's partial
  auto dot = [&](double (*slot)[kMaxGroups], int q, const double* a, int as, const double* b, int bs) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 5; ++k) t = fma(a[k * as], b[k * bs], t);
    if (!own) t = 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) slot[q][grp] = t;
  };
  // the cloth's sum of partials q in `slot`, valid in lane 0: a block is four groups
  auto sum = [&](double (*slot)[kMaxGroups], int q) {
    double s = 0.0;
    if (lane < nblk) {
      double part[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int g = 4 * lane + i, rk = g / groups, lg = g - rk * groups;
        const double* src = slot[q];
        if (CLUSTER) src = cg::this_cluster().map_shared_rank(src, rk < csize ? rk : 0);
        part[i] = rk < csize ? src[lg] : 0.0;
      }
      s = four_sum(part[0], part[1], part[2], part[3]);
    }
    return lanes_sum(s, nblk);
  };
  // two sums to out, a warp each
  auto totals = [&](double (*slot)[kMaxGroups]) {
    if (wid < 2) {
      const double s = sum(slot, wid);
      if (lane == 0) out[wid] = s;
    }
    __syncthreads();
  };

  double held[HOLD ? kRowCoefs : 1];
  if (HOLD && own) {
#pragma unroll
    for (int j = 0; j < kRowCoefs; ++j) held[j] = m < 3 || j < 24 ? coef(j) : 0.0;
  }
  // set-up (k_pcg_setup, k_pcg_start): x = 0, r = b, p = z = D^-1 r
  double x[2] = {0.0, 0.0}, r[2] = {0.0, 0.0}, dinv[2] = {0.0, 0.0};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (i >= nc) break;
    if (own) {
      r[i] = ld(b, m + i, nt, n);
      dinv[i] = ld(so.dinv, m + i, nt, n);
    }
    rs[(m + i) * own_nodes + at] = r[i];
    zs[(m + i) * own_nodes + at] = dinv[i] * r[i];
  }
  for (int e = threadIdx.x; e < WN; e += blockDim.x)
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int64_t g = (int64_t)k * nt + off + win.lo + e;
      sp[k * WN + e] = so.dinv[g] * b[g];
    }
  __syncthreads();
  int red = 0;  // reductions so far: selects the partials' buffer
  if (m == 0) dot(gp[0], 0, rs + at, own_nodes, rs + at, own_nodes);
  if (m == 1) dot(gp[0], 1, rs + at, own_nodes, zs + at, own_nodes);
  sync_all();
  totals(gp[red++ & 1]);
  const double bb = out[0];
  const double thr = pcg_threshold(so.tol, bb);
  double rzc = out[1], rrc = bb;
  bool active = ok_sys && bb != 0.0 && bb >= thr;
  int iters = 0, capped = 0;
  for (int it = 0; it < cap && active; ++it) {
    // q = A p and p.q (k_pcg_spmv)
    double q[2] = {0.0, 0.0};
    if (own) {
      if (HOLD) row_product<TRANS>(m, [&](int j) { return held[HOLD ? j : 0]; }, x_at, q);
      else row_product<TRANS>(m, coef, x_at, q);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (i < nc) rs[(m + i) * own_nodes + at] = q[i];
    if (m == 3 && grp == 0 && lane == 0) irz = 1.0 / rzc;  // by the warp that finishes first
    __syncthreads();
    if (m == 3) dot(gp[red & 1], 0, sp + pos, WN, rs + at, own_nodes);
    sync_all();
    // alpha, by one warp (a division is some ten FP64 instructions, and every
    // warp of the CTA would issue them); x += alpha p, r -= alpha q, |r|^2 and
    // r.z (k_pcg_axpy)
    if (wid == 0) {
      const double pq = sum(gp[red & 1], 0);
      if (lane == 0) out[0] = rzc / pq;
    }
    ++red;
    __syncthreads();
    const double alpha = out[0];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (i >= nc) break;
      if (own) pcg_advance(alpha, sp[(m + i) * WN + pos], q[i], x[i], r[i]);
      rs[(m + i) * own_nodes + at] = r[i];
      zs[(m + i) * own_nodes + at] = dinv[i] * r[i];
    }
    __syncthreads();
    if (m == 0) dot(gp[red & 1], 0, rs + at, own_nodes, rs + at, own_nodes);
    if (m == 1) dot(gp[red & 1], 1, rs + at, own_nodes, zs + at, own_nodes);
    sync_all();
    totals(gp[red++ & 1]);
    // the stop test, then beta and p = z + beta p (k_pcg_dir)
    const double rrn = out[0], rzn = out[1];
    const bool conv = rrn < thr;
    const bool cp = !conv && it + 1 >= maxiter;
    const double beta = rzn * irz;
    rrc = rrn;
    rzc = rzn;
    iters = conv ? it : it + 1;
    if (conv || cp) {
      active = false;
      capped = cp;
      break;
    }
    for (int e = threadIdx.x; e < WN; e += blockDim.x) {
      const int j = win.lo + e, rk = j / own_nodes;
      const double* z = zs + (j - rk * own_nodes);
      if (CLUSTER) z = cg::this_cluster().map_shared_rank(z, rk);
      double zw[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) zw[k] = z[k * own_nodes];
#pragma unroll
      for (int k = 0; k < 5; ++k) sp[k * WN + e] = fma(beta, sp[k * WN + e], zw[k]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (own && i < nc) io.x[rhs * io.x_rhs + (m + i) * io.x_comp + n] = x[i];
  if (rank == 0 && threadIdx.x == 0) {
    pc.bb = bb;
    pc.thr = thr;
    pc.rr = rrc;
    pc.rz[0] = rzc;
    pc.rz[1] = rzc;
    pc.iters = iters;
    pc.active = active ? 1 : 0;
    if (capped) pc.status |= 4;
  }
  // no CTA of the cluster may exit while another can still read its shared memory
  if (CLUSTER) cg::this_cluster().sync();
}

// calls f with the kernel that runs CTAs of up to `groups` groups
template <class F>
cudaError_t with_kernel(int groups, bool cluster, bool trans, F&& f) {
#define YS_PCGC(TT, HOLD)                                                                                     \
  if (groups * 4 * kGroup <= TT) {                                                                            \
    if (cluster) return trans ? f(k_pcg_cluster<TT, true, true, HOLD>) : f(k_pcg_cluster<TT, true, false, HOLD>); \
    return trans ? f(k_pcg_cluster<TT, false, true, HOLD>) : f(k_pcg_cluster<TT, false, false, HOLD>);        \
  }
  YS_PCGC(128, true)
  YS_PCGC(256, false)
  YS_PCGC(512, false)
  YS_PCGC(640, false)
  YS_PCGC(1024, false)
#undef YS_PCGC
  return cudaErrorInvalidValue;
}

void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, const ClusterShape& sh, int ncl, int nrhs) {
  cfg.gridDim = dim3((unsigned)(ncl * sh.csize), (unsigned)nrhs);
  cfg.blockDim = dim3((unsigned)cluster_threads(sh));
  cfg.dynamicSmemBytes = sh.shared;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)sh.csize;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = sh.csize > 1 ? 1 : 0;
}

}  // namespace

// clusters of the shape that fit on the GPU at once; enables its kernels
static cudaError_t cluster_fit(const ClusterShape& sh, int sms, int* clusters) {
  *clusters = 0;
  cudaError_t e = cudaSuccess;
  for (int trans = 0; trans < 2 && e == cudaSuccess; ++trans)
    e = with_kernel(sh.groups, sh.csize > 1, trans != 0, [&](auto* k) {
      cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterShared);
      if (r == cudaSuccess && sh.csize > 8) r = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (r != cudaSuccess) return r;
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1] = {};
      config(cfg, at, sh, 1, 1);
      int fit = 0;
      if (sh.csize > 1) {
        r = cudaOccupancyMaxActiveClusters(&fit, k, &cfg);
      } else {
        r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k, cluster_threads(sh), sh.shared);
        fit *= sms;
      }
      if (r == cudaSuccess) *clusters = trans == 0 || fit < *clusters ? fit : *clusters;
      return r;
    });
  return e;
}

// The groups of a CTA: more of them put a cloth on fewer SMs, which one cloth
// wants least and a batch that fills the GPU most. An iteration takes about
// groups + 2.5 times a group's product (two cluster barriers and the sums), and
// the batch as many rounds of it as it has CTAs per SM, or as its clusters take
// turns. Steps of 17 x 17 cloths in a graph with 1, 2, 3, 5, 8 groups, us (cost):
// one cloth 205, 224, 251, 308, 419 (3.5 to 10.5); 24 cloths 371, 324, 302, 358,
// 467 (10.5, 9, 5.5, 7.5, 10.5); 64 cloths 805, 609, 558, 474, 584 (24, 18, 11,
// 7.5, 10.5); 256 cloths 2880, 2161, 2023, 1682, 2122 (94, 63, 38, 30, 42).
//
// And the schedule: 1.6 us a unit of cost, 2.05 where CTAs take turns, against
// the phases' 16 us an iteration and 0.62 ns a node. Steps in a graph, us,
// persistent / phases: 1 x 5 x 5 173 / 375, 1 x 17 x 17 202 / 473, 24 of them 307
// / 546, 256 1665 / 1855; 1 x 50 x 50 334 / 507, 7 of them 485 / 681, 64 3742 /
// 3215; 1 x 64 x 64 435 / 482, 7 of them 706 / 842, 8 1028 / 939. Over sides of 10
// to 64 and 1 to 256 cloths the persistent PCG was the faster one wherever the
// rule takes it, in graphs and launch by launch; it leaves the phases to some
// batches that it would step up to 8 % faster in a graph (8 x 50 x 50 694 / 747)
// and up to 21 % launch by launch (16 x 50 x 50 1188 / 1443).
cudaError_t pcg_cluster_shape(const ClothParams* cp, int ncloth, int device, ClusterShape* out) {
  ClusterShape best{};
  *out = best;
  int most = 0, sms = 0;
  int64_t nodes = 0;
  for (int c = 0; c < ncloth; ++c) {
    const int n = cp[c].W * cp[c].H;
    most = n > most ? n : most;
    nodes += n;
  }
  if (most > kClusterMaxNodes) return cudaSuccess;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  const int all = (most + kGroup - 1) / kGroup;
  for (int g = (all + kMaxCluster - 1) / kMaxCluster; g <= kMaxGroups; ++g) {
    ClusterShape sh{g, 1, 0, 0.0, false};
    while (sh.csize * g < all) sh.csize *= 2;
    int win = 0, fit = 0;
    for (int c = 0; c < ncloth; ++c)
      for (int r = 0; r < sh.csize; ++r) {
        const int z = Window(r * g * kGroup, g * kGroup, cp[c].W, cp[c].W * cp[c].H).size();
        win = z > win ? z : win;
      }
    sh.shared = (10 * g * kGroup + 5 * win) * (int)sizeof(double);
    if (cluster_fit(sh, sms, &fit) != cudaSuccess || fit < 1) {
      cudaGetLastError();  // this GPU cannot run the shape
      continue;
    }
    const int64_t ctas = (int64_t)ncloth * sh.csize, turns = (ctas + sms - 1) / sms, waves = (ncloth + fit - 1) / fit;
    const int64_t rounds = turns > waves ? turns : waves;
    sh.cost = (double)rounds * (g + 2.5);
    sh.faster = (rounds > 1 ? 2.05 : 1.6) * sh.cost < 16.0 + 0.62e-3 * (double)nodes;
    if (!best.groups || sh.cost < best.cost) best = sh;
  }
  *out = best;
  return cudaSuccess;
}

cudaError_t launch_pcg_cluster(const View& v, const Solver& so, const ClusterRhs& io, int nrhs, const int* cloths,
                               int ncl, const ClusterShape& sh, int cap, cudaStream_t s) {
  return with_kernel(sh.groups, sh.csize > 1, so.trans != 0, [&](auto* k) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1] = {};
    config(cfg, at, sh, ncl, nrhs);
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, k, v, so, io, cloths, cap);
  });
}

}  // namespace ys
