// ys_kernels.cuh -- launch wrappers of the per-step kernels (ys_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "ys_items.cuh"

namespace ys {

// per-cloth Jacobi-PCG bookkeeping (one entry per cloth)
struct PcgCloth {
  double bb;        // |b|^2
  double thr;       // stop when |r|^2 < thr
  double rz[2];     // r.z of the current iterate, double-buffered by parity
  double rr;        // |r|^2 after the last update
  int active;       // 1 while iterating
  int iters;        // completed iterations
  int maxiter;
  int status;       // bit 0: non-finite system, bit 1: non-finite solution, bit 2: iteration cap
};

// Kernels of a chain are launched so that the next one's blocks are set up while
// the last one runs (programmatic dependent launch): each begins by waiting for
// the kernels before it to end (so before any access, and before any return),
// then lets the next be set up. Some 2 us a launch of a kernel of 4 to 8 us:
// steps of 24 ragged cloths 1.15 -> 0.97 ms, a 61 x 83 system 1.11 -> 0.87. In a
// capture they are plain nodes: a graph's own edges were faster (100 x 100 0.68
// ms for 0.71 with programmatic edges). The PCG's product, axpy and direction of
// batches that fill the GPU are not chained (256 cloths 4.93 ms for 4.96); the
// assembly, the PCG's set-up, the update and the sensitivities' kernels are,
// whatever the batch (4.93 ms either way).
__device__ __forceinline__ void chained() {
#if defined(__CUDA_ARCH__)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}
template <class... P, class... A>
inline void chain(void (*k)(P...), dim3 grid, unsigned block, cudaStream_t s, A&&... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute at[1] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cfg.numAttrs = cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone ? 1 : 0;
  // (arguments convert as in a call; an error stays the runtime's last error, which
  // every entry point reads after its launches)
  cudaLaunchKernelEx(&cfg, k, std::forward<A>(a)...);
}

// sum over a warp, the same bits in every lane
__device__ __forceinline__ double cloth_tree(double s) {
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// thread-block partition of the nodes: blocks never straddle two cloths, so
// per-cloth reductions are a fixed-order sum over a contiguous block range
struct Blocks {
  int nblk;
  const int* blk_cloth;   // [nblk]
  const int* blk_node0;   // [nblk] first node
  const int* blk_count;   // [nblk] nodes in the block
  const int* cloth_blk0;  // [ncloth] first block
  const int* cloth_nblk;  // [ncloth]
  bool by_rows;           // products by four warps per 32 nodes (k_pcg_spmv_rows)
};

struct Solver {
  double* x;      // [5][ntot]
  double* r;      // [5][ntot]
  double* p;      // [5][ntot]
  double* q;      // [5][ntot]
  double* dinv;   // [5][ntot]
  double* part;   // [4][nblk] block partial sums, then [nblk][4] group partials of p.q
  PcgCloth* pc;   // [ncloth]
  int* nactive;   // device counter
  double tol;
  int trans;      // 1: solve A^T x = b (the reference-mode tangent solves)
  int* it_base;   // graph mode: iterations completed before this graph body (device), else null
  const int* hold;  // graph mode: when *hold != 0 the solution check and the update leave every cloth
                    // as it was (the learned solve handed the step to Jacobi-PCG), else null
};

constexpr int kBlock = 128;
constexpr int kMaxProducerBlock = 256;  // block size limit of the record producers

// the producers' `threads` (per block, 32..kMaxProducerBlock) does not change results
void launch_geom(const View& v, const int* nodes, int n, cudaStream_t s);
void launch_edge_records(const View& v, const Records& R, cudaStream_t s, int threads = kBlock);
void launch_bend_records(const View& v, const Records& R, cudaStream_t s, int threads = kBlock);
void launch_face_records(const View& v, const Records& R, cudaStream_t s, int threads = kBlock);
// compression, friction (needs every edge and bend record); then, after the
// shear records, the row blocks, b and so.dinv
// the normals, edge and face records, and pc[].status = 0, in one launch
void launch_state_records(const View& v, const Records& R, const int* nodes, int n, PcgCloth* pc, cudaStream_t s);
void launch_cross(const View& v, const Records& R, cudaStream_t s);
void launch_shear_records(const View& v, const Records& R, cudaStream_t s, int threads = kBlock);
void launch_rows(const View& v, const Records& R, const Solver& so, cudaStream_t s);
void launch_pcg_setup(const View& v, const Blocks& b, const Solver& so, cudaStream_t s);
void launch_pcg_spmv(const View& v, const Blocks& b, const Solver& so, cudaStream_t s);
void launch_pcg_axpy(const View& v, const Blocks& b, const Solver& so, int it, cudaStream_t s);
void launch_pcg_dir(const View& v, const Blocks& b, const Solver& so, int it, cudaStream_t s);
void launch_count_active(const View& v, const Solver& so, cudaStream_t s);
void launch_check_solution(const View& v, const Blocks& b, const Solver& so, cudaStream_t s);
// graph mode: *it_base = 0 before the loop; after each body of m iterations
// count the active cloths, advance *it_base by m and set the while node's
// condition to (some cloth active and *it_base < cap)
void launch_graph_loop_begin(const Solver& so, cudaStream_t s);
void launch_graph_loop_tail(const Solver& so, int ncloth, int m, int cap, cudaGraphConditionalHandle h,
                            cudaStream_t s);
void launch_update(const View& v, const Blocks& b, const Solver& so, cudaStream_t s);
// graph mode of the learned solve: *so.hold = 1 if the solve must be redone by
// Jacobi-PCG (an expired tensor-core wait in *err, a breakdown, or the default
// iteration cap when the caller set none; cloths with a non-finite system excepted)
void launch_learned_verdict(const Solver& so, int ncloth, const int* err, int caller_cap, int* hold,
                            cudaStream_t s);
void launch_spmv(const View& v, const double* x, double* y, cudaStream_t s);

// ---- persistent per-cloth PCG (ys_pcg_cluster.cu): one cluster per listed
// cloth runs that cloth's whole solve (set-up included) with at most `cap`
// iterations. Same results as the phase kernels above.
constexpr int kClusterMaxNodes = 4096;  // of a cloth
constexpr int kClusterShared = (5 * kClusterMaxNodes + 10 * 256) * (int)sizeof(double);
struct ClusterShape {
  int groups;   // of 32 nodes in a CTA (0: a cloth of the batch does not fit, or the GPU cannot run any shape)
  int csize;    // CTAs of a cluster
  int shared;   // dynamic shared memory of a CTA
  double cost;  // of an iteration, in units of a group's product
  bool faster;  // than the phases
};
inline int cluster_threads(const ClusterShape& sh) { return 4 * 32 * sh.groups; }  // of a CTA
// the shape for these cloths (host array); enables its kernels, so outside any capture
cudaError_t pcg_cluster_shape(const ClothParams* cp, int ncloth, int device, ClusterShape* out);
// right-hand sides of one launch: rhs k at b + k b_rhs ([5][ntot]), its solution
// at x + k x_rhs with components x_comp apart, its bookkeeping at pc + k ncloth
struct ClusterRhs {
  const double* b;
  double* x;
  PcgCloth* pc;
  int64_t b_rhs, x_rhs, x_comp;
};
cudaError_t launch_pcg_cluster(const View& v, const Solver& so, const ClusterRhs& io, int nrhs, const int* cloths,
                               int ncl, const ClusterShape& sh, int cap, cudaStream_t s);

// state tangents updated by the tangent step (layout [c][kTangents][ntot])
struct TangentState {
  double* dX;
  double* dV;
  double* dUV;
  double* dUVD;
  double* dUVB;
};
// scratch of the tangent step, in units of kTangents * ntot doubles
constexpr int kTangentScratch = 2 * 20 + 2 * 20 + 6 + 4 * 6 + 2;
// after the step's own assembly (records R, values in v): the tangents of the
// normals, compressions and slide indicators, and rt[k][c][ntot] =
// db_k - dA_k q + h dext_k (without dA_k q when v.trunc; dext [kact][ntot][5]
// may be null) for k < kact; returns the number of kernels
int launch_tangent_residual(const View& v, const Records& R, const int* interior, int n_interior, const double* q,
                            double* scratch, const double* dext, int kact, double* rt, cudaStream_t s);
// solution check, then Cloth::update of the state (solution so.x) and its
// tangents (dq, [5][kTangents][ntot])
void launch_update_dual(const View& v, const Blocks& b, const Solver& so, const double* dq, const TangentState& ts,
                        cudaStream_t s);

// ---- reverse-mode step (ys_adjoint.cu)
// state adjoints, component-major: [0] LPos [3][nt], [1] LVel [3][nt],
// [2] EPos [2][nt], [3] EVel [2][nt], [4] EPosBar [2][nt]
struct AdjIO {
  const double* gin[5];  // dL/d(state after the step)
  double* gout[5];       // dL/d(state before the step)
};
// material adjoints: line[p][l] for p = rho, Y, B of line l; cloth[p][c] for
// p = S, mu
struct AdjParamOut {
  double* line[3];
  double* cloth[2];
};
// scratch of the reverse step, in units of ntot doubles
struct AdjSizes {
  int64_t edge, bend, face, shear, cross, normal;
};
constexpr int kAdjCrossFields = 23;
AdjSizes adjoint_sizes();
struct AdjWork {
  const double* lam;        // [5][ntot]
  const double* q;          // [5][ntot], null in the reference mode
  const double* slide_bar;  // [2][ntot]
  double *edge, *bend, *face, *shear, *cross, *normal;
};
void launch_adj_update(const View& v, const AdjIO& io, const double* q, double* qbar, double* slide_bar,
                       cudaStream_t s);
// adds d(lambda . (b - A q) + slide_bar . slide) to io.gout and writes gp, from
// the records R and the normals and compressions of the assembled step (v.trunc
// selects the reference mode); returns the number of kernels
int launch_adj_vjp(const View& v, const Records& R, const AdjWork& w, const int* interior, int n_interior,
                   const AdjIO& io, const double* line_a, const int* line_cloth, const AdjParamOut& gp,
                   cudaStream_t s);
void launch_adj_ext(const View& v, const double* lambda, double* gext, cudaStream_t s);

}  // namespace ys
