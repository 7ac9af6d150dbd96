// Implicit (backward Euler) path: assembly + preconditioned GMRES(m), one persistent
// kernel per chunk of time steps.
//
// Replaces SolverImGPU::update / ::calculate (src/solverIm-gpu.cpp:687-843: Update_HH,
// Update_Mat, Update_B, then BiCGSTAB over cuSPARSE csrmv and cuBLAS dot/axpy with a
// host sync every 30 iterations) and computes the system of SolverImCPU::createMatrix
// (src/solverIm-cpu.cpp:29-183):
//
//   row j (physical):  -g_j V_mother + d_j V_j - g_DR V_DR - b_j g_DL V_DL = rhs_j
//   d_j   = c_j + b_j g_DL + [DR column] g_DR + [mother column] g_j,  c_j = c_m dX/dT - W dX
//   rhs_j = c_m dX V^n_j/dT + K dX + I_j,      g_x = 1/(r_a dX)_x
//
// with the reference's sealed ends: row 1 has no mother column, a row whose next element
// is a terminal has no DR column, and rows 0, N-1 and terminals are identity rows whose
// right-hand side is the stale second buffer -- so they keep their value from two steps
// back, exactly as the CPU reference leaves them.  The matrix is symmetric; it is stored
// as the diagonal plus the per-row conductance to the mother (the value of the (j,
// mother) and (mother, j) entries), which is the reference's CSR without the duplicated
// off-diagonals.  nrt_export_system expands it to the reference's CSR layout.
//
// Solver: right-preconditioned GMRES(m) (Saad), classical Gram-Schmidt, Givens
// rotations.  Each cycle starts from the true FP64 residual b - A x, so in mixed precision
// (FP32 basis, SpMV, orthogonalisation update and preconditioner) every restart is one
// step of iterative refinement.  Inner products and norms: per-thread partial sums in the
// basis precision over the thread's rows, then FP64 across threads and CTAs in a fixed
// order (deterministic, identical in every CTA).  Initial guess: V^n extrapolated
// linearly from V^{n-1}.  In mixed precision with the tree preconditioner a refinement
// cycle is one preconditioned Richardson step, x += M^-1 r (see implicit_one_step), with
// GMRES cycles taking over when a cycle lowers the true residual less than tenfold; that step
// runs in fused passes over the rows (refine.cuh).
//
// Preconditioners: the exact tree factorisation (tree.cuh), an exact tridiagonal solve of
// every unbranched segment piece, Jacobi, or none.
//
// Memory-level parallelism: the row loops keep several rows per thread in flight and
// issue all of a row's independent loads before they use any: a compact per-row flag
// byte replaces the topology record, the neighbours j-1 and j+1 are loaded speculatively
// (the mother is j-1 except on the first row of a DL child), and only the rare rows with
// a far neighbour make a second, dependent load.  The SpMV is fused with up to kG
// Gram-Schmidt products; the update and the norm share a pass.
//
// Three launch shapes from one template:
//  * kGrid  (one tree): a cooperative launch over the whole GPU; rows and windows are split
//    into contiguous per-CTA ranges; grid-wide syncs separate the phases.
//  * kBlock (batches): a persistent block-per-instance scheduler; each CTA takes the next
//    instance (largest first) from an atomic queue and runs all of its steps with
//    __syncthreads only.  kBlock4 is the same with registers for four CTAs on an SM;
//  * kCluster (batches too small to fill the GPU, and small single trees): a cluster of up to
//    eight CTAs per instance, with the cluster's barrier between the phases.
#include <cooperative_groups.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "cvt.cuh"
#include "hh.cuh"
#include "nrt_solver.h"
#include "pdl.cuh"
#include "record.cuh"

namespace cg = cooperative_groups;

namespace nrt {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxPiece = 256;                 // longest segment piece one sweep handles
constexpr int kMaxDots = kMaxRestart + 1;
constexpr int kSumChunks = 8;                  // row chunks of an instance's sums at most (rows_reduce)
constexpr int kTileBytes = 44 * 1024;          // staging of the segment preconditioner
constexpr int kLevels = 128;                   // level offsets kept in shared memory
constexpr int kBlockWalkBytes = 24 * 1024;     // shared memory of a block's walk
constexpr int kWalkBytes = 190 * 1024;         // shared memory of the one-tree launch's walk
constexpr int kClusterWalkBytes = 64 * 1024;   // and of a cluster's
constexpr int kClusterRows = 8 * 1024;         // one tree of at most this many rows: a cluster
constexpr int kRW = 4;                         // tree preconditioner: rows per thread of a window
constexpr int kMaxWin = kThreads * kRW;        // rows of a window at most
constexpr int kU = 4;                          // rows per thread in flight: SpMV + products
constexpr int kV = 4;                          // rows per thread in flight: streaming passes
constexpr int kA = 1;                          // rows per thread in flight: assembly
constexpr int kR = 2;                          // rows per thread in flight: FP64 residual
constexpr int kG = 8;                          // Gram-Schmidt products per pass over the rows

// Per-row flags of the implicit system (ImView::rowf).
enum : uint8_t {
  R_IDENT = 1,   // identity row
  R_UP = 2,      // column at the mother
  R_DOWNR = 4,   // column at DR == j + 1
  R_DOWNL = 8,   // column at DL
  R_FAR = 16,    // the mother is not j - 1 (first row of a DL child)
  R_HH = 32,     // Hodgkin_Huxley element
  R_INP = 64,    // nonzero injected current
};

struct InstStat {
  int64_t iters;
  int32_t last_iters;
  int32_t nonconv;
  double last_res;
  // passes over the rows (GMRES), for bandwidth accounting: FP64 residuals after the one
  // fused into the assembly, preconditioner applications, solution updates, basis
  // vectors read by the Arnoldi steps (sum of j + 1), and Richardson refinement steps
  int64_t residuals, applies, xupdates, basis, rich;
};

struct ImView {
  int64_t ntot;
  int m;             // GMRES restart (BiCGSTAB: sizes the shared work vectors only)
  int krylov;        // NRT_GMRES or NRT_BICGSTAB
  int scheme;        // NRT_BACKWARD_EULER or NRT_CRANK_NICOLSON
  int precond;
  int tol_mode;
  double tol;
  int max_iter;      // per step per instance; 0 -> instance size; < 0 -> assembly only
  double inner_rel;  // a refinement cycle's inner target relative to its starting residual
  int rich;          // refinement cycles start as preconditioned Richardson steps
  int ninst;
  int tile_rows;     // rows per shared-memory tile (segment preconditioner)
  const uint8_t *rowf;
  const double *cmdt;  // c_m dX / dT
  const double *g64;   // 1 / (r_a dX)
  const float *gf;
  const double *wdx64, *kdx64, *inp64;
  double *diag;
  double *rhs;
  void *Wb, *Z, *yv, *pcd, *pcc;  // T-typed workspace
  const int2 *pieces;             // (first row, length) of every segment piece
  const int *tiles;               // piece index where each tile starts (sentinel at end)
  const int *cta_row;             // kGrid: per-CTA row range [cta_row[c], cta_row[c+1])
  const int *cta_win;             // kGrid: per-CTA window range (tree preconditioner)
  const int *cta_tile;            // kGrid: per-CTA tile range
  const int64_t *inst_row;        // per instance first row (ninst + 1)
  const int *inst_tile;           // per instance tile range (ninst + 1)
  const int *order;               // batch: instance processing order
  int *queue;                     // batch: next index into order
  double *partials;               // kGrid: 2 x gridDim x kMaxDots
  InstStat *stats;
  int64_t ld;                     // row-vector stride: ntot rounded up to kRW rows
  const int *inst_n;              // rows of each instance (inst_row holds where they start)
  const int64_t *inst_out;        // where each instance's rows go without the padding
  // exact tree preconditioner (NRT_PRECOND_TREE, tree.cuh): windows, pieces and levels of
  // each instance.  Piece ids are local to the instance, in level order (deepest first).
  void *cdiag;                    // T[ld]: c_j = c_m dX / dT - W dX, written by the assembly
  int win;                        // rows of a window (a multiple of kRW)
  const uint8_t *pfl;             // [ld] row flags: R_IDENT .. R_FAR, P_FIRST, P_LAST
  const uint16_t *wtp;            // [window][win / kRW]: pieces that start in the window before it
  const int *wbase;               // [window] ordinal (row order) of its first piece
  const int *pmap;                // [piece ordinal] -> piece id
  const int4 *plink;              // [piece id]: ids of its children at DR (or the next row) and
                                  // DL and of its parent (-1: none); w: 1 for a one-row piece
  const int *lev_off;             // per instance: the id one past each level's last piece
  const int *inst_win, *inst_piece, *inst_lev;  // [instance + 1] offsets
  int64_t npieces;                // pieces of all instances
  void *pmob;                     // T[4] per piece: its map in the factorisation
  void *pstat;                    // T[4] per piece: B, bL, inv_f beta_f, e_f of the factors
  void *pval;                     // T[4] per piece, two buffers: A, aL, inv_f alpha_f of a solve
  double *pxb;                    // double[2] per piece, two buffers: V of its first, last row
  const double *pgf;              // per piece: FP64 conductance of its first row to the mother
  void *tinv, *te, *tbeta, *talpha;  // T[ld]: 1 / pivot, g / pivot, beta, alpha
  void *tent;                     // T[4] per thread of a window: the map of its piece's later rows
  void *gwalk;                    // walk_bytes per piece: the walk's numbers beyond walk_cap
  int solo;                       // windows are a warp's (tree.cuh)
  int walk_cap;                   // pieces whose walk fits a CTA's shared memory
  int stage_cap;                  // and those whose maps and links fit as well
};

template <typename T>
struct Work {
  T *Wb, *Z, *y, *pd, *pc;
};

struct Shared {
  double *H, *cs, *sn, *g, *s, *y, *red, *warp, *part, *wpart;
  void *coef;      // T[kMaxDots]: update / solution coefficients
  int *flag;       // [0] convergence, [1] queue slot
  void *tile;      // staging area (segment preconditioner) or the tree walk's numbers
};

__host__ __device__ inline size_t shared_fixed_bytes(int m) {
  return sizeof(double) * ((size_t)(m + 1) * m + 2 * m + 2 * (m + 1) + m + kMaxDots +
                           (kWarps + kSumChunks) * kMaxDots + kSumChunks * kWarps * kG + kMaxDots) +
         32;
}

// The dynamic shared memory of the launch.
__device__ __forceinline__ double *dyn_smem() {
  extern __shared__ __align__(16) double nrt_dyn_smem[];
  return nrt_dyn_smem;
}

__device__ Shared carve(double *base, int m) {
  Shared S;
  S.H = base;
  S.cs = S.H + (m + 1) * m;
  S.sn = S.cs + m;
  S.g = S.sn + m;
  S.s = S.g + (m + 1);
  S.y = S.s + (m + 1);
  S.red = S.y + m;
  S.warp = S.red + kMaxDots;
  S.part = S.warp + kWarps * kMaxDots;
  S.wpart = S.part + kSumChunks * kMaxDots;
  S.coef = (void *)(S.wpart + kSumChunks * kWarps * kG);
  S.flag = (int *)((double *)S.coef + kMaxDots);
  S.tile = (void *)((char *)base + ((shared_fixed_bytes(m) + 127) & ~(size_t)127));
  return S;
}

// ---------------------------------------------------------------- groups
//
// The CTAs that step one instance: the CTA itself (kBlock, kBlock4), the whole cooperative launch
// (kGrid), or a thread-block cluster (kCluster).
enum : int { kBlock = 0, kGrid = 1, kCluster = 2, kBlock4 = 3 };
__host__ __device__ constexpr bool one_cta(int mode) { return mode == kBlock || mode == kBlock4; }

__device__ __forceinline__ int cluster_rank() {
  int r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ int cluster_size() {
  int r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

template <int kMode>
__device__ __forceinline__ int group_rank() {
  return kMode == kGrid ? (int)blockIdx.x : kMode == kCluster ? cluster_rank() : 0;
}
template <int kMode>
__device__ __forceinline__ int group_size() {
  return kMode == kGrid ? (int)gridDim.x : kMode == kCluster ? cluster_size() : 1;
}
template <int kMode>
__device__ __forceinline__ void group_sync() {
  if (kMode == kGrid) {
    __threadfence();
    cg::this_grid().sync();
  } else if (kMode == kCluster) {
    __threadfence();  // what other CTAs of the cluster read goes through device memory
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::
                     : "memory");
    __threadfence();
  } else {
    __syncthreads();
  }
}

// Where a group's CTAs leave partial sums (slot: CTA, or chunk of rows): two buffers in turn.
template <int kMode>
__device__ __forceinline__ double *group_partials(double *partials, int parity) {
  if (kMode == kCluster) {
    const int cluster = (int)blockIdx.x / cluster_size();
    return partials + (size_t)kMaxDots * kSumChunks * (2 * cluster + parity);
  }
  return partials + (size_t)kMaxDots * parity * group_size<kMode>();
}

// ---------------------------------------------------------------- reductions

// Reduces the first k register accumulators of every thread over the CTA into out[0..k)
// (FP64, fixed order: warp shuffle tree, then warps in index order).
template <typename T, int kN>
__device__ __forceinline__ void block_reduce(const T (&acc)[kN], int k, double *warp_part,
                                             double *out) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < kN; i++) {
    if (i < k) {
      double v = (double)acc[i];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) warp_part[w * kMaxDots + i] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < k) {
    double s = 0;
    for (int q = 0; q < kWarps; q++) s += warp_part[q * kMaxDots + threadIdx.x];
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

// Completion over the CTAs of a group: per-CTA sums -> global partials -> group sync ->
// every CTA sums all CTAs' partials in the same order.
template <int kMode>
__device__ void group_finish(int k, double *cta_sums, double *partials, int &parity) {
  const int size = group_size<kMode>(), rank = group_rank<kMode>();
  double *buf = group_partials<kMode>(partials, parity);
  parity ^= 1;
  if (threadIdx.x < k) buf[(size_t)rank * kMaxDots + threadIdx.x] = cta_sums[threadIdx.x];
  __syncthreads();
  group_sync<kMode>();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = w; i < k; i += kWarps) {
    double v = 0;
    for (int c = lane; c < size; c += 32) v += buf[(size_t)c * kMaxDots + i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) cta_sums[i] = v;
  }
  __syncthreads();
}

// Sums k accumulators over the group into S.red[off .. off + k).
template <int kMode, typename T, int kN>
__device__ __forceinline__ void group_reduce(const T (&acc)[kN], int k, Shared &S,
                                             double *partials, int &parity, int off = 0) {
  block_reduce(acc, k, S.warp, S.red + off);
  if (!one_cta(kMode)) group_finish<kMode>(k, S.red + off, partials, parity);
}

// ---------------------------------------------------------------- row kernels

// b_r - (A x)_r for the kN rows r = rb + u * stride (rows >= r1 give 0, flag R_IDENT), in
// FP64 as fused multiply-adds: b - d x first (one rounding for the two terms that nearly
// cancel), then + g x_q for each neighbour.  D / G: diagonal and conductance arrays, x the
// vector.  All independent loads of the kN rows are issued before any use.
template <int kN>
__device__ __forceinline__ void residual_rows(const PackView &pv, const ImView &iv,
                                              const double *__restrict__ B,
                                              const double *__restrict__ D,
                                              const double *__restrict__ G, const double *x,
                                              int64_t rb, int64_t stride, int64_t r1,
                                              double (&out)[kN], uint8_t (&fl)[kN]) {
  using C = double;
  using X = double;
  const int64_t N = pv.ntot;
  C dg[kN], gm[kN], gp[kN], bb[kN];
  X xs[kN], xm[kN], xp[kN];
#pragma unroll
  for (int u = 0; u < kN; u++) {
    const int64_t r = rb + u * stride;
    const bool ok = r < r1;
    const int64_t rm = r > 0 ? r - 1 : r, rp = r + 1 < N ? r + 1 : r;
    fl[u] = ok ? iv.rowf[r] : (uint8_t)R_IDENT;
    bb[u] = ok ? B[r] : (C)0;
    dg[u] = ok ? D[r] : (C)0;
    gm[u] = ok ? G[r] : (C)0;
    gp[u] = ok ? G[rp] : (C)0;
    xs[u] = ok ? x[r] : (X)0;
    xm[u] = ok ? x[rm] : (X)0;
    xp[u] = ok ? x[rp] : (X)0;
  }
#pragma unroll
  for (int u = 0; u < kN; u++) {
    const uint8_t f = fl[u];
    X s = 0;
    if (!(f & R_IDENT)) {
      X mo = xm[u], xl = 0;
      C gl = 0;
      if (f & (R_FAR | R_DOWNL)) {
        const Topo t = pv.topo[rb + u * stride];
        if (f & R_FAR) mo = x[t.mother];
        if (f & R_DOWNL) {
          gl = G[t.dl];
          xl = x[t.dl];
        }
      }
      s = fma(-dg[u], xs[u], bb[u]);
      if (f & R_UP) s = fma(gm[u], mo, s);
      if (f & R_DOWNR) s = fma(gp[u], xp[u], s);
      if (f & R_DOWNL) s = fma(gl, xl, s);
    }
    out[u] = s;
  }
}

// (A x)_r in the difference form c_r x_r + sum over the row's neighbours q of
// g_q (x_r - x_q): the same product as apply_rows (the diagonal is c_r plus the row's
// conductances), without its cancellation.  For the smooth vectors of a stiff cable,
// d_r x_r and g x_q are each ~g/c times larger than their difference, so the diagonal
// form loses that factor of precision in FP32; here each difference of neighbouring
// values is formed first (exactly, when they are within a factor of two).
template <int kN, typename C, typename X>
__device__ __forceinline__ void apply_rows_c(const PackView &pv, const ImView &iv,
                                             const C *__restrict__ Cc, const C *__restrict__ G,
                                             const X *x, int64_t rb, int64_t stride, int64_t r1,
                                             X (&out)[kN], uint8_t (&fl)[kN]) {
  const int64_t N = pv.ntot;
  C cc[kN], gm[kN], gp[kN];
  X xs[kN], xm[kN], xp[kN];
#pragma unroll
  for (int u = 0; u < kN; u++) {
    const int64_t r = rb + u * stride;
    const bool ok = r < r1;
    const int64_t rm = r > 0 ? r - 1 : r, rp = r + 1 < N ? r + 1 : r;
    fl[u] = ok ? iv.rowf[r] : (uint8_t)R_IDENT;
    cc[u] = ok ? Cc[r] : (C)0;
    gm[u] = ok ? G[r] : (C)0;
    gp[u] = ok ? G[rp] : (C)0;
    xs[u] = ok ? x[r] : (X)0;
    xm[u] = ok ? x[rm] : (X)0;
    xp[u] = ok ? x[rp] : (X)0;
  }
#pragma unroll
  for (int u = 0; u < kN; u++) {
    const uint8_t f = fl[u];
    X s = 0;
    if (!(f & R_IDENT)) {
      X mo = xm[u], xl = 0;
      C gl = 0;
      if (f & (R_FAR | R_DOWNL)) {
        const Topo t = pv.topo[rb + u * stride];
        if (f & R_FAR) mo = x[t.mother];
        if (f & R_DOWNL) {
          gl = G[t.dl];
          xl = x[t.dl];
        }
      }
      s = cc[u] * xs[u];
      if (f & R_UP) s += gm[u] * (xs[u] - mo);
      if (f & R_DOWNR) s += gp[u] * (xs[u] - xp[u]);
      if (f & R_DOWNL) s += gl * (xs[u] - xl);
    }
    out[u] = s;
  }
}

// ---------------------------------------------------------------- kernel context

template <typename T, int kMode>
struct Ctx {
  // device-memory copies of the launch's views: phases read the fields they need
  const PackView *pv;
  const ImView *iv;
  Work<T> w;
  int64_t r0, r1;   // rows of this CTA in the row passes
  int t0, t1;       // segment-preconditioner tiles
  // tree preconditioner: this CTA's windows, the instance's first and past-the-last window, its first row, the end of
  // its rows (a multiple of kRW after its first), its pieces and level entries
  int w0, w1, iw0, iw1;
  int64_t wrow0, wend;
  int ip0, np, l0, l1;
  int rank;         // this CTA in its group
  int n, chunks, v0, v1;  // rows of the instance; their chunks, this CTA's of them (rows_reduce)
  int wchunks, wv0, wv1;  // chunks of whole windows, this CTA's of them (refine.cuh)
  int wend_of[kSumChunks];  // past the last window of each of this CTA's chunks
  const int *lev;   // the instance's level offsets (in shared memory, when they fit)
};

// The initial guess of a step: V^n extrapolated from V^{n-1} (which Vout holds until the
// first solution update writes it).
__device__ __forceinline__ double x0_of(const double *Vin, const double *Vout, int64_t j) {
  return 2.0 * Vin[j] - Vout[j];
}

// Where a CTA puts the sums of its chunks, kMaxDots apart.
template <int kMode>
__device__ __forceinline__ double *chunk_sums(Shared &S, double *partials, int &parity) {
  if (kMode != kCluster) return S.part;
  parity ^= 1;
  return group_partials<kMode>(partials, parity ^ 1);
}

// The totals of k sums over the instance's chunks, in the order of the chunks, to S.red[off ..], once
// every CTA has put its chunks' (a grid's CTA one, its own).
template <int kMode>
__device__ __forceinline__ void total_chunks(int k, int chunks, const double *sum, Shared &S,
                                             double *partials, int &parity, int off) {
  if (kMode == kGrid) {
    __syncthreads();
    if (threadIdx.x < k) S.red[off + threadIdx.x] = sum[threadIdx.x];
    __syncthreads();
    group_finish<kMode>(k, S.red + off, partials, parity);
    return;
  }
  group_sync<kMode>();
  if (threadIdx.x < k) {
    double s = 0;
    for (int v = 0; v < chunks; v++) s += sum[v * kMaxDots + threadIdx.x];
    S.red[off + threadIdx.x] = s;
  }
  __syncthreads();
}

// Sums k (<= kG) accumulators of a row pass f(first row, end) over the instance into S.red[off .. off + k).  In
// a block or a cluster the rows are taken in up to kSumChunks chunks whose sums are added in
// order, so that the result does not depend on how many CTAs share the instance.  A chunk has 128
// rows or more: four warps keep an SM's FP64 pipe busy, and shorter ones, one after the other,
// only add their latency (1000 cables of 60 compartments in FP64, 32 steps: 20.0 ms with 8 chunks
// each, 6.4 with one).  The warps leave their sums of every chunk and meet once after the last
// (400 trees of 3000: 27.0 -> 25.9 ms).  Where an instance never has more than a CTA (every
// preconditioner but the tree's, and BiCGSTAB) the rows are one chunk: a GMRES cycle of many
// Arnoldi steps reduces up to kG products per pass, and eight short passes took up to three times
// one long one (Jacobi, FP64, 400 trees of 3000, 8 steps: 287 -> 116 ms; mixed, 24 of 3000: 72 -> 32).
template <typename T, int kMode, typename F>
__device__ __forceinline__ void rows_reduce(const Ctx<T, kMode> &c, int k, Shared &S,
                                            double *partials, int &parity, int off, F f) {
  if (kMode == kGrid) {
    auto acc = f(c.r0, c.r1);
    group_reduce<kMode>(acc.v, k, S, partials, parity, off);
    return;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // A chunk of at most 128 rows is one row each for half of the CTA's threads, so the halves take
  // a chunk in turn, the upper one from half a CTA before it (600 cables of 1000 in FP64: 12.3 ->
  // 10.7 ms).  turn: this warp's half, 2 where all warps take every chunk.
  const int turn = c.chunks > 1 && c.n <= kThreads / 2 * c.chunks ? w / (kWarps / 2) : 2;
  for (int v = c.v0; v < c.v1; v++) {  // no barrier between the chunks
    double *to = S.wpart + ((v - c.v0) * kWarps + w) * kG;
    if (turn != 2 && ((v - c.v0) & 1) != turn) {
      if (lane < k) to[lane] = 0.0;
      continue;
    }
    auto acc = f(c.wrow0 + (int64_t)c.n * v / c.chunks - (turn == 1 ? kThreads / 2 : 0),
                 c.wrow0 + (int64_t)c.n * (v + 1) / c.chunks);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(acc.v) / sizeof(acc.v[0])); i++) {
      if (i < k) {
        double x = (double)acc.v[i];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) to[i] = x;
      }
    }
  }
  __syncthreads();
  // the warps' sums of a chunk: eight lanes each
  double *sum = chunk_sums<kMode>(S, partials, parity);
  const int count = (c.v1 - c.v0) * k;
  for (int q0 = 4 * w; q0 < count; q0 += 4 * kWarps) {
    const int q = q0 + (lane >> 3), v = q / k, i = q % k;
    double x = q < count ? S.wpart[(v * kWarps + (lane & 7)) * kG + i] : 0.0;
    for (int o = 4; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o, 8);
    if (q < count && (lane & 7) == 0) sum[(c.v0 + v) * kMaxDots + i] = x;
  }
  total_chunks<kMode>(k, c.chunks, sum, S, partials, parity, off);
}

template <typename X, int kN>
struct Sums {
  X v[kN];
};

}  // namespace nrt

#include "tree.cuh"
#include "refine.cuh"

namespace nrt {

// ---------------------------------------------------------------- segment preconditioner

// Rows covered by tile q: from its first piece's start to its last piece's end.
__device__ __forceinline__ void tile_rows(const ImView &iv, int q, int64_t &a, int64_t &b) {
  const int pa = iv.tiles[q], pb = iv.tiles[q + 1];
  a = iv.pieces[pa].x;
  const int2 last = iv.pieces[pb - 1];
  b = (int64_t)last.x + last.y;
}

// Thomas factorisation of every piece (once per step): pd = 1/pivot, pc = c'.
// Staged through shared memory tile by tile; one thread per piece.
template <typename T, int kMode>
__device__ __noinline__ void factor_pieces(const Ctx<T, kMode> &c) {
  Shared S = carve(dyn_smem(), c.iv->m);
  T *sd = (T *)S.tile;                          // diag, then pivots^-1
  T *sg = sd + c.iv->tile_rows;                  // conductance to the mother
  T *sc = sg + c.iv->tile_rows;                  // c'
  for (int q = c.t0; q < c.t1; q++) {
    int64_t a, b;
    tile_rows(*c.iv, q, a, b);
    for (int64_t r = a + threadIdx.x; r < b; r += blockDim.x) {
      sd[r - a] = (T)c.iv->diag[r];
      sg[r - a] = (T)c.iv->g64[r];
    }
    __syncthreads();
    for (int p = c.iv->tiles[q] + threadIdx.x; p < c.iv->tiles[q + 1]; p += blockDim.x) {
      const int2 pc = c.iv->pieces[p];
      const int o = (int)(pc.x - a);
      double cprev = 0;
      for (int k = 0; k < pc.y; k++) {
        const double sub = k ? -(double)sg[o + k] : 0.0;                  // (j, j-1)
        const double sup = k + 1 < pc.y ? -(double)sg[o + k + 1] : 0.0;   // (j, j+1)
        const double d = 1.0 / ((double)sd[o + k] - sub * cprev);
        cprev = sup * d;
        sd[o + k] = (T)d;
        sc[o + k] = (T)cprev;
      }
    }
    __syncthreads();
    for (int64_t r = a + threadIdx.x; r < b; r += blockDim.x) {
      c.w.pd[r] = sd[r - a];
      c.w.pc[r] = sc[r - a];
    }
    __syncthreads();
  }
}

// z = M^-1 v over this CTA's rows (identity rows: v and z are 0).  eliminated: the tree
// factorisation has eliminated v already.
template <typename T, int kMode>
__device__ __noinline__ void apply_precond(const Ctx<T, kMode> &c, const T *v, T *z,
                                           bool eliminated = false) {
  Shared S = carve(dyn_smem(), c.iv->m);
  if (c.iv->precond == NRT_PRECOND_TREE) {
    group_sync<kMode>();  // v of every row visible (windows hold other threads' and CTAs' rows)
    tree_apply(c, v, z, eliminated);
  } else if (c.iv->precond == NRT_PRECOND_SEGMENT) {
    T *sv = (T *)S.tile;
    T *sd = sv + c.iv->tile_rows;
    T *sc = sd + c.iv->tile_rows;
    T *sg = sc + c.iv->tile_rows;
    for (int q = c.t0; q < c.t1; q++) {
      int64_t a, b;
      tile_rows(*c.iv, q, a, b);
      for (int64_t r = a + threadIdx.x; r < b; r += blockDim.x) {
        sv[r - a] = v[r];
        sd[r - a] = c.w.pd[r];
        sc[r - a] = c.w.pc[r];
        sg[r - a] = (T)c.iv->g64[r];
      }
      __syncthreads();
      for (int p = c.iv->tiles[q] + threadIdx.x; p < c.iv->tiles[q + 1]; p += blockDim.x) {
        const int2 pc = c.iv->pieces[p];
        const int o = (int)(pc.x - a);
        T y = sv[o] * sd[o];
        sv[o] = y;
        for (int k = 1; k < pc.y; k++) {  // forward: y_k = (v_k + g_k y_{k-1}) d_k
          y = (sv[o + k] + sg[o + k] * y) * sd[o + k];
          sv[o + k] = y;
        }
        for (int k = pc.y - 2; k >= 0; k--) {  // backward: z_k = y_k - c'_k z_{k+1}
          y = sv[o + k] - sc[o + k] * y;
          sv[o + k] = y;
        }
      }
      __syncthreads();
      for (int64_t r = a + threadIdx.x; r < b; r += blockDim.x) z[r] = sv[r - a];
      __syncthreads();
    }
  } else {
    for (int64_t j = c.r0 + threadIdx.x; j < c.r1; j += blockDim.x) {
      const uint8_t f = c.iv->rowf[j];
      if (f & R_IDENT) {
        z[j] = 0;
        continue;
      }
      z[j] = c.iv->precond == NRT_PRECOND_JACOBI ? (T)((double)v[j] / c.iv->diag[j]) : v[j];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- one step
//
// The row passes below are separate (not inlined) functions: each keeps its own rows in
// flight in registers, and none of them has to share the register file with the state
// of the others.

template <typename T>
struct DotAcc {
  T v[kG];
};

// Assembly: gates (from V^n), W, K, diagonal, c and right-hand side, fused with the first
// true residual r = b - A x0 (into W_0).  Nothing writes V here, so the neighbours' x0 are
// formed from V^n and V^{n-1} directly (a row's columns are never identity rows).  Returns
// the thread's parts of ||b||^2 and ||r||^2.
template <typename T, int kMode>
__device__ __noinline__ double2 ph_assemble(const Ctx<T, kMode> &c, int64_t r0, int64_t r1, const double *Vin,
                                            const double *Vout, int active, int inst) {
  const PackView &pv = *c.pv;
  const ImView &iv = *c.iv;
  const int64_t N = pv.ntot, stride = blockDim.x;
  T *cdiag = (T *)iv.cdiag;
  // ||b|| needs a few digits only and its terms are far from FP32's range limits: it
  // accumulates in T.  Residual entries near convergence are tiny (their squares leave
  // FP32's normal range), so ||r|| stays in FP64.
  T bacc = 0;
  double racc = 0;
  // gates of this precision (the mixed path keeps them in FP32)
  T *gate = sizeof(T) == 4 ? (T *)(void *)pv.gatef : (T *)(void *)pv.gate;
  const bool cn = iv.scheme == NRT_CRANK_NICOLSON;
  for (int64_t rb = r0 + threadIdx.x; rb < r1; rb += kA * stride) {
    uint8_t f[kA];
    double v[kA], vo[kA], cm[kA], gj[kA], gn[kA], inp[kA], xm[kA], xp[kA], vm[kA], vp[kA];
    int64_t hc[kA];
    T g0[kA], g1[kA], g2[kA];
    // every load that does not depend on the row's flags goes out in this first round
#pragma unroll
    for (int u = 0; u < kA; u++) {
      const int64_t r = rb + u * stride;
      const bool ok = r < r1;
      const int64_t rp = r + 1 < N ? r + 1 : r, rm = r > 0 ? r - 1 : r;
      hc[u] = ok && pv.hp_cls ? (int64_t)pv.hp_cls[r] : (pv.hp_inst ? (int64_t)inst : r);
      const bool gl = ok && pv.hh_dense;
      g0[u] = gl ? gate[r] : (T)0;
      g1[u] = gl ? gate[N + r] : (T)0;
      g2[u] = gl ? gate[2 * N + r] : (T)0;
      f[u] = ok ? iv.rowf[r] : (uint8_t)R_IDENT;
      v[u] = ok ? Vin[r] : 0.0;
      vo[u] = ok ? Vout[r] : 0.0;
      cm[u] = ok ? iv.cmdt[r] : 0.0;
      gj[u] = ok ? iv.g64[r] : 0.0;
      gn[u] = ok ? iv.g64[rp] : 0.0;
      inp[u] = 0.0;
      xm[u] = ok ? x0_of(Vin, Vout, rm) : 0.0;
      xp[u] = ok ? x0_of(Vin, Vout, rp) : 0.0;
      vm[u] = ok && cn ? Vin[rm] : 0.0;  // Crank-Nicolson: V^n of the neighbours
      vp[u] = ok && cn ? Vin[rp] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kA; u++) {
      const int64_t r = rb + u * stride;
      if (r >= r1) continue;
      double wdx, kdx;
      if (f[u] & R_HH) {
        const int64_t L = pv.hp_ld;
        if (!pv.hh_dense) {
          g0[u] = gate[r];
          g1[u] = gate[N + r];
          g2[u] = gate[2 * N + r];
        }
        if (sizeof(T) == 4) {
          const HHParams32 q = hh_params32(pv.hpq, hc[u]);
          const float dv = (float)(v[u] - (double)q.v[HP_REST]);
          GateStep32 g = hh_step32(dv + q.v[HP_LSNA], dv + q.v[HP_LSK], (float)g0[u],
                                   (float)g1[u], (float)g2[u], q.v[HP_DTMS], q.v[HP_GNA],
                                   q.v[HP_GK], q.v[HP_GL], q.v[HP_ENA], q.v[HP_EK], q.v[HP_EL]);
          gate[r] = (T)g.m;
          gate[N + r] = (T)g.h;
          gate[2 * N + r] = (T)g.n;
          const float dx = q.v[HP_DX];
          wdx = (double)(g.W * dx);  // FP32 inputs: the product in FP32 loses nothing
          kdx = (double)(g.K * dx);
        } else {
          const double *hp = pv.hp + hc[u];
          GateStep64 g = hh_step64(v[u], (double)g0[u], (double)g1[u], (double)g2[u],
                                   hp[HP_LSNA * L], hp[HP_LSK * L], hp[HP_REST * L],
                                   hp[HP_DTMS * L], hp[HP_GNA * L], hp[HP_GK * L],
                                   hp[HP_GL * L], hp[HP_ENA * L], hp[HP_EK * L],
                                   hp[HP_EL * L]);
          gate[r] = (T)g.m;
          gate[N + r] = (T)g.h;
          gate[2 * N + r] = (T)g.n;
          const double dx = hp[HP_DX * L];
          wdx = g.W * dx;
          kdx = g.K * dx;
        }
      } else {
        wdx = iv.wdx64[r];
        kdx = iv.kdx64[r];
      }
      if (f[u] & R_IDENT) {
        c.w.y[r] = 0;
        c.w.Wb[r] = 0;
        continue;
      }
      // backward Euler: c = c_m dX/dT - W dX; Crank-Nicolson (doubled): 2 c_m dX/dT - W dX
      const double cj = (cn ? 2.0 * cm[u] : cm[u]) - wdx;
      double d = cj, gl = 0.0, xl = 0.0, xmo = xm[u], vmo = vm[u], vl = 0.0;
      if (f[u] & (R_DOWNL | R_FAR)) {
        const Topo t = pv.topo[r];
        if (f[u] & R_DOWNL) {
          gl = iv.g64[t.dl];
          xl = x0_of(Vin, Vout, t.dl);
          if (cn) vl = Vin[t.dl];
          d += gl;
        }
        if (f[u] & R_FAR) {
          xmo = x0_of(Vin, Vout, t.mother);
          if (cn) vmo = Vin[t.mother];
        }
      }
      if (f[u] & R_DOWNR) d += gn[u];
      if (f[u] & R_UP) d += gj[u];
      iv.diag[r] = d;
      cdiag[r] = (T)cj;
      if (active && (f[u] & R_INP)) inp[u] = iv.inp64[r];  // one row or a few per tree
      double b;
      if (!cn) {
        b = cm[u] * v[u] + kdx;
        if (active && (f[u] & R_INP)) b += inp[u];  // other rows would add an exact 0
      } else {  // (2 c_m dX/dT + W dX) V^n - sum g (V^n - V^n_q) + 2 (K dX + I)
        b = (2.0 * cm[u] + wdx) * v[u];
        if (f[u] & R_UP) b -= gj[u] * (v[u] - vmo);
        if (f[u] & R_DOWNR) b -= gn[u] * (v[u] - vp[u]);
        if (f[u] & R_DOWNL) b -= gl * (v[u] - vl);
        b += 2.0 * kdx;
        if (active && (f[u] & R_INP)) b += 2.0 * inp[u];
      }
      iv.rhs[r] = b;
      bacc += (T)b * (T)b;
      // r = b - A x0 as residual_rows forms it: b - d x0, then mother, DR, DL
      double rr = fma(-d, 2.0 * v[u] - vo[u], b);
      if (f[u] & R_UP) rr = fma(gj[u], xmo, rr);
      if (f[u] & R_DOWNR) rr = fma(gn[u], xp[u], rr);
      if (f[u] & R_DOWNL) rr = fma(gl, xl, rr);
      c.w.Wb[r] = (T)rr;
      racc += rr * rr;
    }
  }
  return make_double2((double)bacc, racc);
}

// Vout = x0 for the rows of this group (when a step ends before any solution update).
template <typename T, int kMode>
__device__ __noinline__ void ph_x0(const Ctx<T, kMode> &c, const double *Vin, double *Vout) {
  const uint8_t *rowf = c.iv->rowf;
  for (int64_t j = c.r0 + threadIdx.x; j < c.r1; j += blockDim.x)
    if (!(rowf[j] & R_IDENT)) Vout[j] = x0_of(Vin, Vout, j);
}

// True residual r = b - A x in FP64 into W_0 (identity rows 0); returns the thread's
// part of ||r||^2, or with scale > 0 of ||scale r||^2 summed in FP32.  That form is for
// the mixed GMRES and Richardson cycles, where the norm only decides convergence and scales
// an FP32 basis: it keeps the sum off the FP64 pipe, and the caller passes a power of two
// near 1 / (the previous residual norm), which keeps the entries in FP32's range.  FP64
// solves and BiCGSTAB (whose rho_0 is this norm squared) take the FP64 sum.
template <typename T, int kMode>
__device__ __noinline__ double ph_residual(const Ctx<T, kMode> &c, int64_t r0, int64_t r1, const double *x, float scale) {
  const PackView &pv = *c.pv;
  const ImView &iv = *c.iv;
  const int64_t stride = blockDim.x;
  float acc = 0;
  double acc64 = 0;
  for (int64_t rb = r0 + threadIdx.x; rb < r1; rb += kR * stride) {
    double rr[kR];
    uint8_t fl[kR];
    residual_rows<kR>(pv, iv, iv.rhs, iv.diag, iv.g64, x, rb, stride, r1, rr, fl);
#pragma unroll
    for (int u = 0; u < kR; u++) {
      const int64_t r = rb + u * stride;
      if (r >= r1) continue;
      if (fl[u] & R_IDENT) {
        c.w.Wb[r] = 0;
        continue;
      }
      c.w.Wb[r] = (T)rr[u];
      if (scale > 0) {
        const float e = (float)rr[u] * scale;
        acc = fmaf(e, e, acc);
      } else {
        acc64 += rr[u] * rr[u];
      }
    }
  }
  return scale > 0 ? (double)acc : acc64;
}

// y = s_j A Z_j, fused with the thread's parts of <y, W_i> for i < g1.
template <typename T, int kMode>
__device__ __noinline__ DotAcc<T> ph_spmv(const Ctx<T, kMode> &c, int64_t r0, int64_t r1, int j, T sj, int g1) {
  const PackView &pv = *c.pv;
  const ImView &iv = *c.iv;
  const int64_t ld = iv.ld, stride = blockDim.x;
  const T *CT = (const T *)iv.cdiag;
  const T *GT = sizeof(T) == 4 ? (const T *)(const void *)iv.gf : (const T *)(const void *)iv.g64;
  const T *Zj = c.w.Z + (size_t)j * ld;
  DotAcc<T> acc;
#pragma unroll
  for (int i = 0; i < kG; i++) acc.v[i] = 0;
  for (int64_t rb = r0 + threadIdx.x; rb < r1; rb += kU * stride) {
    T y[kU];
    uint8_t fl[kU];
    apply_rows_c<kU>(pv, iv, CT, GT, Zj, rb, stride, r1, y, fl);
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int64_t r = rb + u * stride;
      y[u] *= sj;
      if (r < r1) c.w.y[r] = y[u];
    }
#pragma unroll
    for (int i = 0; i < kG; i++) {
      if (i < g1) {
        const T *Wi = c.w.Wb + (size_t)i * ld;
#pragma unroll
        for (int u = 0; u < kU; u++) {
          const int64_t r = rb + u * stride;
          if (r < r1) acc.v[i] += y[u] * Wi[r];
        }
      }
    }
  }
  return acc;
}

// The thread's parts of <y, W_{i0+i}> for i < gk.
template <typename T, int kMode>
__device__ __noinline__ DotAcc<T> ph_products(const Ctx<T, kMode> &c, int64_t r0, int64_t r1, int i0, int gk) {
  const int64_t ld = c.iv->ld, stride = blockDim.x;
  DotAcc<T> acc;
#pragma unroll
  for (int i = 0; i < kG; i++) acc.v[i] = 0;
  for (int64_t rb = r0 + threadIdx.x; rb < r1; rb += kV * stride) {
    T y[kV];
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t r = rb + u * stride;
      y[u] = r < r1 ? c.w.y[r] : (T)0;
    }
#pragma unroll
    for (int i = 0; i < kG; i++) {
      if (i < gk) {
        const T *Wi = c.w.Wb + (size_t)(i0 + i) * ld;
#pragma unroll
        for (int u = 0; u < kV; u++) {
          const int64_t r = rb + u * stride;
          if (r < r1) acc.v[i] += y[u] * Wi[r];
        }
      }
    }
  }
  return acc;
}

// W_{j+1} = y - sum_{i <= j} coef_i W_i; returns the thread's part of ||W_{j+1}||^2.
template <typename T, int kMode>
__device__ __noinline__ T ph_update(const Ctx<T, kMode> &c, int64_t r0, int64_t r1, int j, const T *coef) {
  const int64_t ld = c.iv->ld, stride = blockDim.x;
  T *Wn = c.w.Wb + (size_t)(j + 1) * ld;
  T nacc = 0;
  for (int64_t rb = r0 + threadIdx.x; rb < r1; rb += kV * stride) {
    T a[kV];
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t r = rb + u * stride;
      a[u] = r < r1 ? c.w.y[r] : (T)0;
    }
#pragma unroll 1
    for (int i = 0; i <= j; i++) {
      const T ci = coef[i];
      const T *Wi = c.w.Wb + (size_t)i * ld;
      T w[kV];
#pragma unroll
      for (int u = 0; u < kV; u++) {
        const int64_t r = rb + u * stride;
        w[u] = r < r1 ? Wi[r] : (T)0;
      }
#pragma unroll
      for (int u = 0; u < kV; u++) a[u] -= ci * w[u];
    }
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t r = rb + u * stride;
      if (r < r1) {
        Wn[r] = a[u];
        nacc += a[u] * a[u];
      }
    }
  }
  return nacc;
}

// V += sum_{i < k} coef_i Z_i (identity rows keep their value).  With Vin non-null this is
// the step's first update and V starts from x0 = 2 Vin - V.
template <typename T, int kMode>
__device__ __noinline__ void ph_xupdate(const Ctx<T, kMode> &c, int k, const T *coef, double *Vout,
                                        const double *Vin) {
  const int64_t ld = c.iv->ld, stride = blockDim.x;
  const uint8_t *rowf = c.iv->rowf;
  for (int64_t rb = c.r0 + threadIdx.x; rb < c.r1; rb += kV * stride) {
    T a[kV];
    uint8_t fl[kV];
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t r = rb + u * stride;
      a[u] = 0;
      fl[u] = r < c.r1 ? rowf[r] : (uint8_t)R_IDENT;
    }
#pragma unroll 1
    for (int i = 0; i < k; i++) {
      const T ci = coef[i];
      const T *Zi = c.w.Z + (size_t)i * ld;
      T z[kV];
#pragma unroll
      for (int u = 0; u < kV; u++) {
        const int64_t r = rb + u * stride;
        z[u] = r < c.r1 ? Zi[r] : (T)0;
      }
#pragma unroll
      for (int u = 0; u < kV; u++) a[u] += ci * z[u];
    }
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t r = rb + u * stride;
      if (!(fl[u] & R_IDENT)) {
        const double base = Vin ? x0_of(Vin, Vout, r) : Vout[r];
        Vout[r] = base + (double)a[u];
      }
    }
  }
}

// ---- BiCGSTAB (right-preconditioned, on the correction equation of one refinement cycle)

// p = r + beta (p - omega v); beta == 0 gives p = r.
template <typename T, int kMode>
__device__ __noinline__ void ph_bicg_dir(const Ctx<T, kMode> &c, const T *r, T *p, const T *v, T beta,
                                         T omega) {
  const int64_t stride = blockDim.x;
  for (int64_t rb = c.r0 + threadIdx.x; rb < c.r1; rb += kV * stride) {
    T a[kV], b[kV], d[kV];
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t q = rb + u * stride;
      const bool ok = q < c.r1;
      a[u] = ok ? r[q] : (T)0;
      b[u] = ok && beta != (T)0 ? p[q] : (T)0;
      d[u] = ok && beta != (T)0 ? v[q] : (T)0;
    }
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t q = rb + u * stride;
      if (q < c.r1) p[q] = a[u] + beta * (b[u] - omega * d[u]);
    }
  }
}

// out = A x; returns the thread's parts of <out, d0> and <out, d1> (d1 may be null).
template <typename T, int kMode>
__device__ __noinline__ DotAcc<T> ph_matvec(const Ctx<T, kMode> &c, const T *x, T *out, const T *d0,
                                            const T *d1) {
  const PackView &pv = *c.pv;
  const ImView &iv = *c.iv;
  const int64_t stride = blockDim.x;
  const T *CT = (const T *)iv.cdiag;
  const T *GT = sizeof(T) == 4 ? (const T *)(const void *)iv.gf : (const T *)(const void *)iv.g64;
  DotAcc<T> acc;
#pragma unroll
  for (int i = 0; i < kG; i++) acc.v[i] = 0;
  for (int64_t rb = c.r0 + threadIdx.x; rb < c.r1; rb += kU * stride) {
    T y[kU], e0[kU], e1[kU];
    uint8_t fl[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int64_t q = rb + u * stride;
      e0[u] = q < c.r1 ? d0[q] : (T)0;
      e1[u] = q < c.r1 && d1 ? d1[q] : (T)0;
    }
    apply_rows_c<kU>(pv, iv, CT, GT, x, rb, stride, c.r1, y, fl);
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int64_t q = rb + u * stride;
      if (q < c.r1) out[q] = y[u];
      acc.v[0] += y[u] * e0[u];
      acc.v[1] += y[u] * e1[u];
    }
  }
  return acc;
}

// s = r - alpha v; returns the thread's part of ||s||^2.
template <typename T, int kMode>
__device__ __noinline__ T ph_bicg_s(const Ctx<T, kMode> &c, const T *r, const T *v, T alpha, T *s) {
  const int64_t stride = blockDim.x;
  T acc = 0;
  for (int64_t rb = c.r0 + threadIdx.x; rb < c.r1; rb += kV * stride) {
    T a[kV], b[kV];
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t q = rb + u * stride;
      a[u] = q < c.r1 ? r[q] : (T)0;
      b[u] = q < c.r1 ? v[q] : (T)0;
    }
#pragma unroll
    for (int u = 0; u < kV; u++) {
      const int64_t q = rb + u * stride;
      const T x = a[u] - alpha * b[u];
      if (q < c.r1) s[q] = x;
      acc += x * x;
    }
  }
  return acc;
}

// V += alpha ph + omega sh (FP64 accumulation; identity rows keep their value) and
// r = s - omega t; returns the thread's parts of ||r||^2 and <rh, r>.
template <typename T, int kMode>
__device__ __noinline__ DotAcc<T> ph_bicg_x(const Ctx<T, kMode> &c, const T *ph, const T *sh,
                                            const T *s, const T *t, T alpha, T omega, T *r,
                                            const T *rh, double *Vout) {
  const int64_t stride = blockDim.x;
  const uint8_t *rowf = c.iv->rowf;
  DotAcc<T> acc;
#pragma unroll
  for (int i = 0; i < kG; i++) acc.v[i] = 0;
  for (int64_t rb = c.r0 + threadIdx.x; rb < c.r1; rb += kU * stride) {
    T a[kU], b[kU], e[kU], f[kU], h[kU];
    uint8_t fl[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int64_t q = rb + u * stride;
      const bool ok = q < c.r1;
      a[u] = ok ? ph[q] : (T)0;
      b[u] = ok ? sh[q] : (T)0;
      e[u] = ok ? s[q] : (T)0;
      f[u] = ok ? t[q] : (T)0;
      h[u] = ok ? rh[q] : (T)0;
      fl[u] = ok ? rowf[q] : (uint8_t)R_IDENT;
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int64_t q = rb + u * stride;
      const T rn = e[u] - omega * f[u];
      if (q < c.r1) r[q] = rn;
      if (!(fl[u] & R_IDENT)) Vout[q] += (double)(alpha * a[u] + omega * b[u]);
      acc.v[0] += rn * rn;
      acc.v[1] += rn * h[u];
    }
  }
  return acc;
}

// One refinement cycle of BiCGSTAB on A d = r0 (r0 in W_0, ||r0|| = res), accumulating
// d into V.  Stops at the cycle target, at the budget, or on a breakdown (the next cycle
// restarts from the true residual).  Every pass through the loop counts against the
// budget, so repeated breakdowns still end the step.
// Not inlined, so that the GMRES path's register allocation does not carry it.
// Returns {parity, iters}.
template <typename T, int kMode>
__device__ __noinline__ int2 bicgstab_cycle(const Ctx<T, kMode> &c, int parity, double res,
                                            double cycle_target, int budget, int iters,
                                            double *Vout) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const int64_t ld = iv.ld;
  T *rh = c.w.Wb, *r1 = c.w.Wb + ld, *p = c.w.Wb + 2 * ld, *v = c.w.Wb + 3 * ld;
  T *ph = c.w.Z, *sh = c.w.Z + ld, *s = c.w.Z + 2 * ld, *t = c.w.Z + 3 * ld;
  const T *r = rh;  // the first iteration reads r0 itself
  double rho = res * res, rho_prev = 1.0, alpha = 1.0, omega = 1.0;
  for (int it = 0; iters < budget; it++) {
    const double beta = it == 0 ? 0.0 : (rho / rho_prev) * (alpha / omega);
    ph_bicg_dir(c, r, p, v, (T)beta, (T)omega);
    group_sync<kMode>();
    apply_precond(c, p, ph);
    group_sync<kMode>();
    {
      DotAcc<T> acc = ph_matvec(c, ph, v, rh, (const T *)nullptr);
      group_reduce<kMode>(acc.v, 1, S, iv.partials, parity);
    }
    const double rv = S.red[0];
    if (rv == 0.0 || !(rv == rv) || !(rho == rho)) {  // breakdown: restart from r0
      iters++;
      break;
    }
    alpha = rho / rv;
    {
      T acc[1] = {ph_bicg_s(c, r, v, (T)alpha, s)};
      group_reduce<kMode>(acc, 1, S, iv.partials, parity);
    }
    iters++;
    if (sqrt(S.red[0]) <= cycle_target) {  // x += alpha ph completes the cycle
      ph_bicg_x(c, ph, ph, s, s, (T)alpha, (T)0, r1, rh, Vout);
      group_sync<kMode>();
      break;
    }
    apply_precond(c, s, sh);
    group_sync<kMode>();
    {
      DotAcc<T> acc = ph_matvec(c, sh, t, s, t);
      group_reduce<kMode>(acc.v, 2, S, iv.partials, parity);
    }
    const double ts = S.red[0], tt = S.red[1];
    omega = tt > 0.0 ? ts / tt : 0.0;
    {
      DotAcc<T> acc = ph_bicg_x(c, ph, sh, s, t, (T)alpha, (T)omega, r1, rh, Vout);
      group_reduce<kMode>(acc.v, 2, S, iv.partials, parity);
    }
    r = r1;
    const double rn = sqrt(S.red[0]);
    rho_prev = rho;
    rho = S.red[1];
    if (rn <= cycle_target || omega == 0.0 || rho == 0.0) break;
  }
  group_sync<kMode>();  // V complete before the next true residual
  return make_int2(parity, iters);
}

// One backward-Euler step of one group (CTA or grid) for instance `inst`.
template <typename T, int kMode>
__device__ __forceinline__ void implicit_one_step(const Ctx<T, kMode> &c, Shared &S, int &parity, const double *Vin,
                                                  double *Vout, bool active, int64_t inst_n,
                                                  int inst) {
  const ImView &iv = *c.iv;
  const int m = iv.m;
  T *coef = (T *)S.coef;
  // ---- assembly, fused with the first true residual (W_0); V still holds V^{n-1}
  const bool tree = iv.precond == NRT_PRECOND_TREE;
  const bool fused = sizeof(T) == 4 && iv.rich != 0;  // by windows, with the pieces' matrices
  double target = iv.tol, res0 = 0;
  auto assemble = [&](int64_t r0, int64_t r1) {
    const double2 br = ph_assemble(c, r0, r1, Vin, Vout, active ? 1 : 0, inst);
    return Sums<double, 2>{{br.x, br.y}};
  };
  if (fused) {
    if constexpr (sizeof(T) == 4) {
      if (iv.scheme == NRT_CRANK_NICOLSON)
        refine_assemble<kMode, true>(c, Vin, Vout, active ? 1 : 0, inst);
      else
        refine_assemble<kMode, false>(c, Vin, Vout, active ? 1 : 0, inst);
      sum_windows<kMode, 2>(c, S, iv.partials, parity);  // also publishes W_0, the matrices
    }
  } else {
    rows_reduce(c, 2, S, iv.partials, parity, 0, assemble);  // also publishes W_0 and c
  }
  if (iv.tol_mode == NRT_TOL_REL) target = iv.tol * sqrt(S.red[0]);
  res0 = sqrt(S.red[1]);
  __syncthreads();  // S.red is read before the next sum
  if (iv.precond == NRT_PRECOND_SEGMENT) {
    factor_pieces(c);
  } else if (tree && !fused) {
    tree_maps(c);
    group_sync<kMode>();
  }
  if (tree) tree_factor(c, c.w.Wb, fused);
  const int budget = iv.max_iter > 0 ? iv.max_iter : (iv.max_iter < 0 ? 0 : (int)inst_n);
  const double inner_rel = iv.inner_rel;
  int iters = 0, n_res = 0, n_app = 0, n_xup = 0, n_basis = 0, n_rich = 0;
  double res = 0, prev_res = 0;
  bool converged = false;
  bool x0_pending = true;  // V holds V^{n-1} until the first solution update
  bool rich_done = false;  // the last cycle's update has left the true residual in res
  bool w0_valid = true;    // W_0 holds the residual
  int pb = 0;              // the buffer of the pieces' values that the next walk reads
  bool eliminated = tree;  // the right-hand side W_0 has been eliminated
  // Mixed precision with the tree preconditioner: M is the FP32 factorisation of A itself,
  // so GMRES's one Arnoldi step per cycle takes x += y M^-1 r with y within rounding of 1.
  // A Richardson step takes x += M^-1 r without the SpMV, the products and the basis
  // update.  The FP64 residual that opens the next cycle checks it: a cycle that does not
  // lower the true residual tenfold hands the rest of the step to GMRES cycles.
  bool rich = iv.rich != 0;
  for (int cycle = 0;; cycle++) {
    // ---- cycle start: true residual r = b - A x in FP64, W_0 = r, Z_0 = M^-1 r
    if (cycle == 0) {
      res = res0;
    } else if (!rich_done) {
      // res > 0 here (a zero residual has converged); the scale stays a normal FP32 number
      const bool f32 = sizeof(T) == 4 && iv.krylov == NRT_GMRES;
      const int e = f32 ? max(-126, min(126, ilogb(res))) : 0;
      const float scale = f32 ? pow2_of<float>(-e) : 0.0f;
      rows_reduce(c, 1, S, iv.partials, parity, 0, [&](int64_t r0, int64_t r1) {
        return Sums<double, 1>{{ph_residual(c, r0, r1, Vout, scale)}};
      });
      res = sqrt(S.red[0]) * pow2_of<double>(e);
      n_res++;
    }
    rich_done = false;
    if (res <= target) {
      converged = true;
      break;
    }
    if (iters + n_rich >= budget || !(res == res)) break;  // budget spent, or not finite
    if (rich && cycle > 0 && res > 0.1 * prev_res) rich = false;
    if (iv.krylov == NRT_BICGSTAB) {
      if (x0_pending) {
        ph_x0(c, Vin, Vout);
        x0_pending = false;
        group_sync<kMode>();
      }
      const int2 pi = bicgstab_cycle(c, parity, res, fmax(target, inner_rel * res), budget,
                                     iters, Vout);
      parity = pi.x;
      iters = pi.y;
      continue;
    }
    if constexpr (sizeof(T) == 4) {
      if (rich) {  // x += M^-1 r and the residual of the new x
        if (!eliminated) tree_eliminate(c, c.w.Wb, pb, Vout);
        group_sync<kMode>();  // every window's elimination visible to the walk
        if (walks(c, iv)) refine_walk(c, pb);
        if (!one_cta(kMode) && c.np > iv.walk_cap) group_sync<kMode>();
        const int e = max(-126, min(126, ilogb(res)));
        const float scale = pow2_of<float>(-e);
        // The first cycle's residual is eliminated at once: it is rarely the last.
        if (cycle == 0) {
          pb ^= 1;
          refine_update<kMode, true>(c, Vout, scale, pb);
        } else {
          refine_update<kMode, false>(c, Vout, scale, pb);
        }
        eliminated = cycle == 0;
        sum_windows<kMode, 1>(c, S, iv.partials, parity);  // V and W_0 complete
        prev_res = res;
        res = sqrt(S.red[0]) * pow2_of<double>(e);
        w0_valid = cycle != 0;
        rich_done = true;
        x0_pending = false;
        n_app++;
        n_xup++;
        n_rich++;
        n_res++;
        continue;
      }
    }
    if (!w0_valid) {  // after the first refinement cycle W_0 is not stored
      (void)ph_residual(c, c.r0, c.r1, Vout, 1.0f);
      w0_valid = true;
    }
    apply_precond(c, c.w.Wb, c.w.Z, eliminated && cycle == 0);
    n_app++;
    eliminated = false;
    group_sync<kMode>();  // Z_0 of every row visible before the SpMV
    if (threadIdx.x == 0) {
      S.g[0] = res;
      for (int i = 1; i <= m; i++) S.g[i] = 0;
      S.s[0] = 1.0 / res;
    }
    __syncthreads();
    const double cycle_target = fmax(target, inner_rel * res);
    int k = 0;
    for (int j = 0; j < m; j++) {
      // y = s_j A Z_j fused with p_i = <y, W_i> for the first kG of i <= j
      const int g1 = min(j + 1, kG);
      {
        rows_reduce(c, g1, S, iv.partials, parity, 0,
                    [&](int64_t r0, int64_t r1) { return ph_spmv(c, r0, r1, j, (T)S.s[j], g1); });
      }
      for (int i0 = kG; i0 <= j; i0 += kG) {  // remaining products, kG at a time
        const int gk = min(j + 1 - i0, kG);
        rows_reduce(c, gk, S, iv.partials, parity, i0,
                    [&](int64_t r0, int64_t r1) { return ph_products(c, r0, r1, i0, gk); });
      }
      if (threadIdx.x <= j) {
        const double h = S.s[threadIdx.x] * S.red[threadIdx.x];
        S.H[threadIdx.x * m + j] = h;
        coef[threadIdx.x] = (T)(h * S.s[threadIdx.x]);
      }
      __syncthreads();
      // w = y - sum_i h_ij s_i W_i -> W_{j+1}; ||w||^2
      rows_reduce(c, 1, S, iv.partials, parity, 0, [&](int64_t r0, int64_t r1) {
        return Sums<T, 1>{{ph_update(c, r0, r1, j, coef)}};  // publishes W_{j+1}
      });
      if (threadIdx.x == 0) {
        const double hn = sqrt(S.red[0]);
        S.s[j + 1] = hn > 0 ? 1.0 / hn : 0.0;
        for (int i = 0; i < j; i++) {
          const double a = S.H[i * m + j], b = S.H[(i + 1) * m + j];
          S.H[i * m + j] = S.cs[i] * a + S.sn[i] * b;
          S.H[(i + 1) * m + j] = -S.sn[i] * a + S.cs[i] * b;
        }
        const double a = S.H[j * m + j];
        const double den = sqrt(a * a + hn * hn);
        S.cs[j] = den == 0 ? 1.0 : a / den;
        S.sn[j] = den == 0 ? 0.0 : hn / den;
        S.H[j * m + j] = den;
        S.g[j + 1] = -S.sn[j] * S.g[j];
        S.g[j] = S.cs[j] * S.g[j];
        S.flag[0] = (fabs(S.g[j + 1]) <= cycle_target || hn == 0) ? 1 : 0;
      }
      __syncthreads();
      k = j + 1;
      iters++;
      n_basis += j + 1;
      if (S.flag[0] || iters + n_rich >= budget || k >= m) break;
      // Z_{j+1} = M^-1 W_{j+1}, only when another Arnoldi step will use it
      apply_precond(c, c.w.Wb + (size_t)(j + 1) * iv.ld, c.w.Z + (size_t)(j + 1) * iv.ld);
      n_app++;
      group_sync<kMode>();  // Z_{j+1} of every row visible before the next SpMV
    }
    // ---- x += sum_i y_i s_i Z_i
    if (threadIdx.x == 0) {
      for (int i = k - 1; i >= 0; i--) {
        double a = S.g[i];
        for (int l = i + 1; l < k; l++) a -= S.H[i * m + l] * S.y[l];
        S.y[i] = a / S.H[i * m + i];
      }
      for (int i = 0; i < k; i++) coef[i] = (T)(S.y[i] * S.s[i]);
    }
    __syncthreads();
    ph_xupdate(c, k, coef, Vout, x0_pending ? Vin : (const double *)nullptr);
    group_sync<kMode>();
    n_xup++;
    x0_pending = false;
  }
  if (x0_pending) ph_x0(c, Vin, Vout);  // converged (or out of budget) at x0 itself
  if (threadIdx.x == 0 && c.rank == 0) {
    InstStat &st = iv.stats[inst];
    st.iters += iters;
    st.last_iters = iters;
    st.last_res = res;
    if (!converged) st.nonconv += 1;
    st.residuals += n_res;
    st.applies += n_app;
    st.xupdates += n_xup;
    st.basis += n_basis;
    st.rich += n_rich;
  }
  group_sync<kMode>();  // V^{n+1} complete before the next step reads it
}

// Recording at the probes of instance `inst` after the step at loop index i (V is that
// step's output, complete in this CTA's view).  Each thread keeps the same probes for the
// whole launch.
__device__ __noinline__ void ph_record(const RecView *rp, int inst, int64_t i, const double *V,
                                       double dT) {
  const RecView r = *rp;
  const int a = r.p0[inst], b = r.p0[inst + 1];
  for (int p = a + threadIdx.x; p < b; p += blockDim.x) record_probe(r, p, i, V[r.src[p]], dT);
}

// Resident CTAs per SM that the registers allow.  FP32: 3 (80 registers; the 2048-tree batch
// took 51.1 ms per 8 steps at 4, whose 64 registers spill in the fused passes, 41.7 at 3 and
// 48.9 at 2).  FP64: 2 (128 registers): its FP64 pipe is full with 16 warps.  kBlock4: 4, for the
// batches that four_per_sm names.
template <typename T, int kMode>
constexpr int ctas_per_sm() {
  return kMode == kBlock4 ? 4 : sizeof(T) == 4 ? 3 : 2;
}

template <typename T, int kMode>
__global__ void __launch_bounds__(kThreads, ctas_per_sm<T, kMode>()) implicit_steps(const PackView *pvp, const ImView *ivp,
                                                           int nsteps, int force, double *V0,
                                                           double *V1, int cur,
                                                           const RecView *rec) {
  // The views and the context live in shared memory: the passes read their fields all the time,
  // and from device memory (or the stack) those reads were evicted from L1 by the rows that
  // stream through it.
  __shared__ PackView s_pv;
  __shared__ ImView s_iv;
  __shared__ Ctx<T, kMode> c;
  __shared__ int s_lev[kLevels];
  static_assert(sizeof(PackView) % 4 == 0 && sizeof(ImView) % 4 == 0, "copied by words");
  for (int u = threadIdx.x; u < (int)(sizeof(PackView) / 4); u += kThreads)
    ((int *)&s_pv)[u] = ((const int *)pvp)[u];
  for (int u = threadIdx.x; u < (int)(sizeof(ImView) / 4); u += kThreads)
    ((int *)&s_iv)[u] = ((const int *)ivp)[u];
  __syncthreads();
  const ImView &iv = s_iv;
  Shared S = carve(dyn_smem(), iv.m);
  int parity = 0;
  if (threadIdx.x == 0) {
    c.pv = &s_pv;
    c.iv = &s_iv;
    c.w.Wb = (T *)iv.Wb;
    c.w.Z = (T *)iv.Z;
    c.w.y = (T *)iv.yv;
    c.w.pd = (T *)iv.pcd;
    c.w.pc = (T *)iv.pcc;
    c.rank = group_rank<kMode>();
  }
  __syncthreads();
  const int gsize = group_size<kMode>();
  int q = kMode == kCluster ? (int)blockIdx.x / gsize : 0;
  for (;;) {
    int inst = 0;
    if (one_cta(kMode)) {
      if (threadIdx.x == 0) S.flag[1] = atomicAdd(iv.queue, 1);
      __syncthreads();
      q = S.flag[1];
      __syncthreads();
    }
    if (kMode != kGrid) {
      if (q >= iv.ninst) break;
      inst = iv.order[q];
    }
    const int n = iv.inst_n[inst];
    const bool tree = iv.precond == NRT_PRECOND_TREE;
    if (threadIdx.x == 0) {
      c.n = n;
      c.chunks = tree && iv.krylov == NRT_GMRES ? min(kSumChunks, (n + 127) / 128) : 1;
      c.v0 = c.chunks * c.rank / gsize;
      c.v1 = c.chunks * (c.rank + 1) / gsize;
      c.wrow0 = iv.inst_row[inst];
      c.wend = c.wrow0 + ((n + kRW - 1) & ~(kRW - 1));
      c.r0 = c.wrow0 + (int64_t)n * c.v0 / c.chunks;
      c.r1 = c.wrow0 + (int64_t)n * c.v1 / c.chunks;
      c.iw0 = tree ? iv.inst_win[inst] : 0;
      c.iw1 = tree ? iv.inst_win[inst + 1] : 0;
      c.w0 = c.iw0 + (c.iw1 - c.iw0) * c.rank / gsize;
      c.w1 = c.iw0 + (c.iw1 - c.iw0) * (c.rank + 1) / gsize;
      // gsize divides kSumChunks, so a CTA's windows are whole chunks
      c.wchunks = min(kSumChunks, c.iw1 - c.iw0);
      c.wv0 = c.wchunks * c.rank / gsize;
      c.wv1 = c.wchunks * (c.rank + 1) / gsize;
      for (int v = c.wv0; v < c.wv1; v++) c.wend_of[v - c.wv0] = c.iw0 + (c.iw1 - c.iw0) * (v + 1) / c.wchunks;
      c.ip0 = tree ? iv.inst_piece[inst] : 0;
      c.np = tree ? iv.inst_piece[inst + 1] - c.ip0 : 0;
      c.l0 = tree ? iv.inst_lev[inst] : 0;
      c.l1 = tree ? iv.inst_lev[inst + 1] : 0;
      if (kMode == kGrid) {
        c.r0 = iv.cta_row[blockIdx.x];
        c.r1 = iv.cta_row[blockIdx.x + 1];
        c.t0 = iv.cta_tile[blockIdx.x];
        c.t1 = iv.cta_tile[blockIdx.x + 1];
        if (tree) {
          c.w0 = iv.cta_win[blockIdx.x];
          c.w1 = iv.cta_win[blockIdx.x + 1];
          c.wchunks = c.wv1 = 1;
          c.wv0 = 0;
          c.wend_of[0] = c.w1;
        }
      } else {
        c.t0 = iv.inst_tile[inst];
        c.t1 = iv.inst_tile[inst + 1];
      }
    }
    __syncthreads();
    // a walk reads its level offsets level by level: from shared memory
    const int nlev = c.l1 - c.l0;
    for (int u = threadIdx.x; u < nlev && nlev <= kLevels; u += kThreads) s_lev[u] = iv.lev_off[c.l0 + u];
    if (threadIdx.x == 0) c.lev = nlev <= kLevels ? s_lev : iv.lev_off + c.l0;
    __syncthreads();
    if (tree) stage_links(c);
    const InstDev in = s_pv.inst[inst];
    int s = 0;
    for (; s < nsteps; s++) {
      const int64_t i = in.base + s;
      if (i >= in.iend) break;
      const bool active = force >= 0 ? force != 0 : (i >= in.ion && i <= in.ioff);
      implicit_one_step<T, kMode>(c, S, parity, ((cur + s) & 1) ? V1 : V0,
                                  ((cur + s + 1) & 1) ? V1 : V0, active, n, inst);
      if (rec && c.rank == 0) ph_record(rec, inst, i, ((cur + s + 1) & 1) ? V1 : V0, in.dT);
    }
    if ((nsteps - s) & 1) {  // the run ended inside the launch: its latest V goes where the
      double *dst = ((cur + nsteps) & 1) ? V1 : V0;  // others' is, each CTA moving its rows
      const double *src = ((cur + s) & 1) ? V1 : V0;
      for (int64_t j = c.r0 + threadIdx.x; j < c.r1; j += blockDim.x) dst[j] = src[j];
    }
    if (kMode == kGrid) break;
    if (kMode == kCluster) q += (int)gridDim.x / gsize;
    group_sync<kMode>();
  }
}

// ---------------------------------------------------------------- host side

// Windows, pieces and levels of the exact tree preconditioner (tree.cuh), per instance and
// then concatenated.
struct TreePlan {  // sized without a fill: every entry is written by the builder
  hvec<uint8_t> pfl;
  hvec<uint16_t> wtp;
  hvec<int> wbase, pmap, lev_off, inst_win, inst_piece, inst_lev;
  hvec<int4> plink;
  hvec<double> pgf;
  int max_pieces = 0;
};

struct ImplicitState {
  ImView iv{};
  PackView *d_pv = nullptr;  // device copies the kernel reads
  ImView *d_iv = nullptr;
  hvec<uint8_t> rowf;  // sized without a fill: implicit_plan writes every row
  hvec<int2> pieces;
  std::vector<int> tiles, cta_row, cta_tile, cta_win, inst_tile, order, inst_n;
  std::vector<int64_t> inst_row;
  TreePlan tree;
  int grid_blocks = 0;
  bool grid_mode = false;
  int cluster = 0;  // CTAs per cluster (0: not a cluster launch)
  int win = 0;      // rows per window of the tree preconditioner
  int tile_rows = 0;
  size_t smem = 0;
  const void *kern = nullptr;
};

static const void *implicit_kernel(bool mixed, int group) {
  if (mixed)
    return group == kGrid ? (const void *)implicit_steps<float, kGrid>
           : group == kCluster ? (const void *)implicit_steps<float, kCluster>
           : group == kBlock4 ? (const void *)implicit_steps<float, kBlock4>
                              : (const void *)implicit_steps<float, kBlock>;
  return group == kGrid ? (const void *)implicit_steps<double, kGrid>
         : group == kCluster ? (const void *)implicit_steps<double, kCluster>
         : group == kBlock4 ? (const void *)implicit_steps<double, kBlock4>
                            : (const void *)implicit_steps<double, kBlock>;
}

static size_t smem_bytes(int m, size_t tile) {
  return ((shared_fixed_bytes(m) + 127) & ~(size_t)127) + tile;
}

// Takes room for max(count, room) entries and uploads count of them (src may be null).
template <typename X>
static int up(Arena &a, X *&dst, const X *src, size_t count, cudaStream_t st, size_t room = 1) {
  dst = (X *)a.take(sizeof(X) * std::max(count, room));
  if (!dst) {
    set_error("arena exhausted");
    return NRT_ENOMEM;
  }
  if (src && count) NRT_CUDA(cudaMemcpyAsync(dst, src, sizeof(X) * count, cudaMemcpyHostToDevice, st));
  return NRT_OK;
}

#define TRYI(x)                     \
  do {                              \
    int _rc = (x);                  \
    if (_rc != NRT_OK) return _rc;  \
  } while (0)

// One instance's pieces: runs of rows linked to the row before them (mother == j - 1),
// broken after branch points, at identity rows and at window edges.  A piece's parent row
// (the mother of its first row) is always the last row of another piece.  Level = number of
// pieces above it; ids count the pieces level by level, deepest level first.
struct InstPieces {
  std::vector<int> wbase, pmap, lev_off;
  std::vector<int4> plink;
  std::vector<double> pgf;
};

static void instance_pieces(const HostPack &host, const uint8_t *rowf, int32_t i, int win,
                            uint8_t *pfl, uint16_t *wtp, InstPieces &L) {
  struct Piece {
    int parent, level, c1, c2;
    int64_t row;
    int len;
  };
  const int64_t o = host.off[i], n = host.num_elem[i];
  const int64_t n4 = (n + kRW - 1) & ~(int64_t)(kRW - 1), nw = (n + win - 1) / win;
  constexpr uint8_t keep = R_IDENT | R_UP | R_DOWNR | R_DOWNL | R_FAR;
  std::vector<Piece> pc;
  std::vector<int> piece_of(n, -1);
  L.wbase.resize(nw);
  int cur = -1, max_level = -1;
  for (int64_t j = 0; j < nw * win; j++) {
    if (j % win == 0) L.wbase[j / win] = (int)pc.size();
    if (j % kRW == 0)
      wtp[(j / win) * (win / kRW) + (j % win) / kRW] = (uint16_t)(pc.size() - L.wbase[j / win]);
    if (j >= n) {
      if (j < n4) pfl[j] = P_IDENT;
      continue;
    }
    const uint8_t f = rowf[j] & keep;
    pfl[j] = f;
    if (f & R_IDENT) {
      cur = -1;
      continue;
    }
    const bool linked = cur >= 0 && j % win != 0 && (f & R_UP) && !(f & R_FAR) &&
                        !(host.topo[o + j - 1].flags & F_BRANCH);
    if (!linked) {
      const int64_t m = (f & R_UP) ? host.topo[o + j].mother - o : -1;
      Piece p{m >= 0 ? piece_of[m] : -1, 0, -1, -1, o + j, 0};
      if (p.parent >= 0) {
        p.level = pc[p.parent].level + 1;
        Piece &q = pc[p.parent];
        (q.c1 < 0 ? q.c1 : q.c2) = (int)pc.size();
      }
      max_level = std::max(max_level, p.level);
      pc.push_back(p);
      cur = (int)pc.size() - 1;
      pfl[j] |= P_FIRST;
    }
    piece_of[j] = cur;
    pc[cur].len++;
    // the piece ends here unless the next row continues it
    const bool more = j + 1 < n && (j + 1) % win != 0 && !(rowf[j + 1] & R_IDENT) &&
                      (rowf[j + 1] & R_UP) && !(rowf[j + 1] & R_FAR) &&
                      !(host.topo[o + j].flags & F_BRANCH);
    if (!more) pfl[j] |= P_LAST;
  }
  const int np = (int)pc.size(), nl = max_level + 1;
  std::vector<int> at(nl + 1, 0);
  for (const Piece &p : pc) at[max_level - p.level + 1]++;  // deepest level first
  for (int e = 0; e < nl; e++) at[e + 1] += at[e];
  L.lev_off.assign(at.begin() + 1, at.end());
  L.pmap.resize(np);
  L.plink.resize(np);
  for (int q = 0; q < np; q++) L.pmap[q] = at[max_level - pc[q].level]++;
  auto id = [&](int q) { return q >= 0 ? L.pmap[q] : -1; };
  L.pgf.resize(np);
  for (int q = 0; q < np; q++) {
    L.plink[L.pmap[q]] = make_int4(id(pc[q].c1), id(pc[q].c2), id(pc[q].parent), pc[q].len == 1);
    L.pgf[L.pmap[q]] = host.gax[pc[q].row];
  }
}

static void build_tree_plan(const HostPack &host, const uint8_t *rowf, int64_t ld, int win,
                            TreePlan &T) {
  const int32_t ni = host.ninst;
  std::vector<InstPieces> loc(ni);
  T.inst_win.resize(ni + 1);
  T.inst_piece.resize(ni + 1);
  T.inst_lev.resize(ni + 1);
  T.inst_win[0] = T.inst_piece[0] = T.inst_lev[0] = 0;
  for (int32_t i = 0; i < ni; i++)
    T.inst_win[i + 1] = T.inst_win[i] + (host.num_elem[i] + win - 1) / win;
  T.pfl.resize(ld);
  T.wtp.resize((size_t)T.inst_win[ni] * (win / kRW));
  parallel_for(ni, [&](int64_t i) {
    instance_pieces(host, rowf + host.off[i], (int32_t)i, win, T.pfl.data() + host.off[i],
                    T.wtp.data() + (size_t)T.inst_win[i] * (win / kRW), loc[i]);
  });
  for (int32_t i = 0; i < ni; i++) {
    T.inst_piece[i + 1] = T.inst_piece[i] + (int)loc[i].pmap.size();
    T.inst_lev[i + 1] = T.inst_lev[i] + (int)loc[i].lev_off.size();
    T.max_pieces = std::max(T.max_pieces, (int)loc[i].pmap.size());
  }
  T.wbase.resize(T.inst_win[ni]);
  T.pmap.resize(T.inst_piece[ni]);
  T.plink.resize(T.inst_piece[ni]);
  T.pgf.resize(T.inst_piece[ni]);
  T.lev_off.resize(T.inst_lev[ni]);
  parallel_for(ni, [&](int64_t i) {
    const InstPieces &L = loc[i];
    std::copy(L.wbase.begin(), L.wbase.end(), T.wbase.begin() + T.inst_win[i]);
    std::copy(L.pmap.begin(), L.pmap.end(), T.pmap.begin() + T.inst_piece[i]);
    std::copy(L.plink.begin(), L.plink.end(), T.plink.begin() + T.inst_piece[i]);
    std::copy(L.pgf.begin(), L.pgf.end(), T.pgf.begin() + T.inst_piece[i]);
    std::copy(L.lev_off.begin(), L.lev_off.end(), T.lev_off.begin() + T.inst_lev[i]);
  });
}

// Groups pieces [pa, pb) into tiles whose row span fits the shared-memory staging area.
static void make_tiles(const hvec<int2> &pieces, int pa, int pb, int tile_rows,
                       std::vector<int> &tiles) {
  int64_t start_row = -1;
  for (int p = pa; p < pb; p++) {
    const int64_t end = (int64_t)pieces[p].x + pieces[p].y;
    if (start_row < 0 || end - start_row > tile_rows) {
      tiles.push_back(p);
      start_row = pieces[p].x;
    }
  }
}

// Whether a batch of one CTA per tree runs kBlock4 (the same results: a tree's arithmetic and its
// order are the same in both).
//
// With 64 registers instead of 80 (mixed) or 128 (FP64) a CTA's passes take longer, and a batch lasts
// as long as its largest tree's CTA does (1000 trees of 1e3 to 3e4: mixed 9.6 ms, 12.0 with four;
// 2048 of 1e3 to 1e5 34.9 and 39.6).  Four are as fast or faster where the number of trees decides:
//  - trees that are too small to occupy a CTA's warps, more than the usual CTAs take at once (32
//    steps of 1000 cables of 60: FP64 6.3 ms, 3.9 with four; mixed 2.7, 2.4; of 300: 11.4, 10.0 and
//    3.2, 2.8);
//  - more trees of about one size than the usual CTAs take at once, when four CTAs need no more
//    rounds' time.  A round of k CTAs per SM lasts as long as k trees on an SM even where it is not
//    full (the trees of the last one meet on few SMs), except that a launch of fewer trees than
//    places spreads them evenly: 400 cables of 3000 in FP64 are two rounds of two, 28.9 ms, or three
//    at once, 21.0; 600 of 1000 mixed two rounds of three, 3.6, or four at once, 2.6; but 620 of
//    1500 mixed two rounds of three, 2.6, or of four, 2.9;
//  - so many trees that the largest, on a quarter of an SM, is done in three quarters of the time
//    that all take: 4096 trees of 1e3 to 1e5 mixed 69.5 ms, 68.9 with four, cables 65.0 and 62.7;
//    3000 cables of 100 to 1000 mixed 2.51 and 2.35; 1500 of 1000 to 3000 in FP64 13.4 and 12.6.
static bool four_per_sm(const HostPack &host, const nrt_options &opt, int sms) {
  const int usual = opt.precision == NRT_MIXED ? ctas_per_sm<float, kBlock>() : ctas_per_sm<double, kBlock>();
  if (opt.tile_ctas_per_sm > 0) return opt.tile_ctas_per_sm > usual;
  const int64_t ni = host.ninst;
  int64_t largest = 0, sum = 0;
  for (int64_t i = 0; i < ni; i++) {
    largest = std::max<int64_t>(largest, host.num_elem[i]);
    sum += host.num_elem[i];
  }
  if (ni <= usual * (int64_t)sms) return false;
  auto trees_per_sm = [&](int64_t k) {
    return ni <= k * sms ? (ni + sms - 1) / sms : (ni + k * sms - 1) / (k * sms) * k;
  };
  return largest <= 512 || (4 * largest * ni <= 5 * sum && trees_per_sm(4) <= trees_per_sm(usual)) ||
         16 * largest * sms <= 3 * sum;
}

static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// Row structure, launch shape and preconditioner schedule; the exact device bytes the
// implicit workspace takes from the arena.
int Engine::implicit_plan(size_t &bytes) {
  im = new ImplicitState();
  ImplicitState &S = *im;
  const int64_t N = host.ntot;
  const int32_t ni = host.ninst;
  // Row structure (flags) per element.  The validator guaranteed the reference
  // numbering: mother < j, DR == j + 1 off terminals, terminals follow their mother.
  S.rowf.resize(N);
  static_assert(kRowAlign == kRW, "instances start on whole row groups");
  parallel_for(ni, [&](int64_t i) {
    const int64_t o = host.off[i], n = host.num_elem[i];
    for (int64_t jl = 0; jl < n; jl++) {
      const int64_t j = o + jl;
      Topo &t = host.topo[j];
      t.flags &= ~(uint32_t)(F_UP | F_DOWNR | F_DOWNL | F_IDENT);
      uint8_t rf = (t.flags & F_HH) ? R_HH : 0;
      if (host.inp[j] != 0.0) rf |= R_INP;
      const bool ident = jl == 0 || jl == n - 1 || (t.flags & F_TERM);
      if (ident) {
        t.flags |= F_IDENT;
        S.rowf[j] = rf | R_IDENT;
        continue;
      }
      if (jl != 1) {
        t.flags |= F_UP;
        rf |= R_UP;
        if (t.mother != j - 1) rf |= R_FAR;
      }
      if (!(host.topo[j + 1].flags & F_TERM)) {  // j + 1 is in this instance (j < o + n - 1)
        t.flags |= F_DOWNR;
        rf |= R_DOWNR;
      }
      if (t.flags & F_BRANCH) {
        t.flags |= F_DOWNL;
        rf |= R_DOWNL;
      }
      S.rowf[j] = rf;
    }
    for (int64_t j = o + n; j < host.off[i + 1]; j++) S.rowf[j] = R_IDENT;  // padding
  });
  S.inst_row.assign(host.off.begin(), host.off.end());
  S.inst_n.assign(host.num_elem.begin(), host.num_elem.end());
  // Segment pieces (segment preconditioner): maximal runs of consecutive physical rows
  // linked to their predecessor (mother == j - 1 with a mother column), cut at kMaxPiece rows.
  const bool tree = opt.precond == NRT_PRECOND_TREE, segs = opt.precond == NRT_PRECOND_SEGMENT;
  std::vector<int> inst_piece(ni + 1, 0);
  if (segs) {
    std::vector<std::vector<int2>> ip(ni);  // per instance, then concatenated in order
    parallel_for(ni, [&](int64_t i) {
      const int64_t o = host.off[i], n = host.num_elem[i];
      int64_t start = -1;
      for (int64_t jl = 0; jl < n; jl++) {
        const int64_t j = o + jl;
        const Topo &t = host.topo[j];
        const bool ident = t.flags & F_IDENT;
        const bool linked = !ident && (t.flags & F_UP) && t.mother == j - 1 && start >= 0 &&
                            (j - start) < kMaxPiece;
        if (!linked && start >= 0) {
          ip[i].push_back(make_int2((int)start, (int)(j - start)));
          start = -1;
        }
        if (!ident && start < 0) start = j;
      }
      if (start >= 0) ip[i].push_back(make_int2((int)start, (int)(o + n - start)));
    });
    for (int32_t i = 0; i < ni; i++) inst_piece[i + 1] = inst_piece[i] + (int)ip[i].size();
    S.pieces.resize(inst_piece[ni]);
    parallel_for(ni, [&](int64_t i) {
      std::copy(ip[i].begin(), ip[i].end(), S.pieces.begin() + inst_piece[i]);
    });
  }
  const int np = (int)S.pieces.size();
  const bool mixed = opt.precision == NRT_MIXED;
  const size_t tb = mixed ? 4 : 8;
  const int64_t ld = (N + kRW - 1) & ~(int64_t)(kRW - 1);
  int64_t max_n = 0;
  for (int32_t i = 0; i < ni; i++) max_n = std::max<int64_t>(max_n, host.num_elem[i]);
  // rows staged at a time: no more than a tree has, so that small trees' CTAs fit an SM
  S.tile_rows = (int)std::min<int64_t>(kTileBytes / (4 * tb), (max_n + 31) & ~(int64_t)31);
  S.tile_rows = std::max(S.tile_rows, kMaxPiece);
  int dev_sms = 0;
  NRT_CUDA(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, device));
  S.grid_mode = ni == 1 && opt.schedule == 0;
  // Clusters (tree preconditioner with GMRES): an instance's rows and windows split over 2, 4 or
  // 8 CTAs, as many as leave every cluster resident at once.  One CTA per instance leaves SMs
  // idle as long as there are fewer instances than SMs, and a small single tree spends most of a
  // cooperative launch's step in its grid-wide syncs (1.5 to 2 us each; a cluster's barrier
  // takes about 0.4).
  S.cluster = 0;
  if (tree && opt.krylov == NRT_GMRES && opt.schedule == 0) {
    // No more CTAs than gain by it, since their barriers cost more than a CTA's: FP64 one per
    // chunk of 128 rows, mixed batches one per window, and a mixed single tree of one window stays
    // with one CTA (32 steps: of 300 compartments 1.76 ms on 4 CTAs, 1.31 on one; of 1000 1.78 on
    // 8, 1.65 on one; of 2000 1.75 on 8, 2.02 on 2; 48 of 300 2.21 ms on 8 CTAs each, 1.33 on one).
    const int64_t part = mixed && (ni > 1 || max_n <= kMaxWin) ? kMaxWin : 128;
    const int64_t parts = (max_n + part - 1) / part;
    int64_t per = mixed ? ctas_per_sm<float, kCluster>() : ctas_per_sm<double, kCluster>();
    if (opt.tile_ctas_per_sm > 0) per = std::min<int64_t>(per, opt.tile_ctas_per_sm);
    const int64_t room = ni > 1 ? dev_sms * per / ni : max_n <= kClusterRows ? 8 : 0;
    for (int cs = 2; cs <= 8 && cs <= room && cs < 2 * parts; cs *= 2) S.cluster = cs;
    if (room && parts == 1) S.grid_mode = false;
  }
  if (S.cluster) S.grid_mode = false;
  if (tree) {
    // Rows per window: 1024, a CTA's.  In an FP64 batch 128, a warp's: its passes lose their
    // barriers, a cluster's CTAs share a tree evenly, and the longer chains of pieces cost less
    // (48 trees of 1e3 to 1e4, 8 steps: 2.50 -> 2.31 ms; 1000 of 300: 5.83 -> 5.18).  The mixed step
    // does not gain: with its warps apart in its longer code 2048 trees of 1e3 to 1e5 took 43.0 ms
    // instead of 37.8.  In a single tree fewer than 1024 (down to 128) where its CTAs
    // would otherwise not all have a window: a window's FP64 arithmetic is bound by its SM's
    // FP64 pipe, so a small tree's windows go to as many SMs as it has CTAs.  (The windows set
    // the order of the scans' sums, so those of a batch do not depend on its size.)
    S.iv.solo = ni > 1 && !mixed;
    S.win = S.iv.solo ? 128 : kMaxWin;
    if (ni == 1) {
      const int64_t ctas = S.cluster ? S.cluster : S.grid_mode ? dev_sms : 1;
      while (S.win > 128 && S.win * ctas >= 2 * max_n) S.win /= 2;
    }
    build_tree_plan(host, S.rowf.data(), ld, S.win, S.tree);
  }
  const int group = S.cluster ? kCluster : S.grid_mode ? kGrid
                    : four_per_sm(host, opt, dev_sms) ? kBlock4 : kBlock;
  const void *kern = implicit_kernel(mixed, group);
  S.kern = kern;
  // shared memory: the segment preconditioner's staging, or the tree walk's numbers of
  // every piece: up to kBlockWalkBytes, which keeps three CTAs on an SM, in a cluster
  // kClusterWalkBytes, or in the one-tree launch, whose CTAs then have an SM each, up to
  // kWalkBytes; larger walks run in device memory.  A block stages the maps and links too where
  // they fit as well (1000 trees of 300 compartments, mixed, 32 steps: 6.03 -> 5.34 ms).
  size_t tile = 0;
  if (segs) tile = (size_t)S.tile_rows * 4 * tb;
  if (tree) {
    const bool grp = !one_cta(group);
    const size_t cap = S.grid_mode ? kWalkBytes : S.cluster ? kClusterWalkBytes : kBlockWalkBytes;
    S.iv.walk_cap = (int)std::min<size_t>(std::min<size_t>(cap / walk_bytes(tb, grp), kNoPiece - 1),
                                          (size_t)S.tree.max_pieces);
    S.iv.stage_cap = grp ? S.iv.walk_cap : (int)std::min<size_t>(cap / walk_bytes(tb, true), S.tree.max_pieces);
    tile = std::max(S.iv.walk_cap * walk_bytes(tb, grp), S.iv.stage_cap * walk_bytes(tb, true));
  }
  S.smem = smem_bytes(opt.restart, tile);
  // The limit is the function's, not the handle's: all that a CTA can have, so that handles
  // of any size launch in any order.
  int smem_limit = 0;
  cudaFuncAttributes fa;
  NRT_CUDA(cudaDeviceGetAttribute(&smem_limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
  NRT_CUDA(cudaFuncGetAttributes(&fa, kern));
  smem_limit -= (int)fa.sharedSizeBytes;
  NRT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_limit));
  int per_sm = 0;
  NRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, S.smem));
  if (per_sm < 1) {
    set_error("implicit kernel does not fit on an SM");
    return NRT_EDEVICE;
  }
  if (S.grid_mode) {
    // One tree: a cooperative grid.  Segment preconditioner: row ranges aligned with its
    // pieces.  Otherwise the row passes and the windows are each split evenly: the rows over
    // as many CTAs as leave each kRowsPerCta (FP64: an SM evaluates one HH row in about 60
    // cycles of its FP64 pipe, so small trees gain from every SM), the windows over the same
    // CTAs as far as they go.  With the tree preconditioner one CTA per SM: a second repeats the
    // walk and lengthens the syncs (100k compartments, per step: mixed 130 -> 113 us, FP64 186 ->
    // 156; the depth-10 binary tree 119 and 212 either way), and it keeps other streams' trees
    // off the GPU (64 served requests: 7.8 -> 6.6 s).
    const int64_t rows_per_cta = segs ? 4 * kThreads : (mixed ? 256 : 64);
    const int64_t want = (N + rows_per_cta - 1) / rows_per_cta;
    int G = (int)std::min<int64_t>((int64_t)dev_sms * (tree ? 1 : std::min(per_sm, 2)), std::max<int64_t>(1, want));
    G = std::max(1, std::min(G, 4096));
    S.cta_row.assign(G + 1, (int)N);
    S.cta_tile.assign(G + 1, 0);
    S.cta_win.assign(G + 1, 0);
    if (segs) {
      std::vector<int> cta_piece(G + 1, np);
      int q = 0;
      for (int c = 0; c < G; c++) {
        const int64_t goal = (N * (int64_t)c) / G;
        while (q < np && S.pieces[q].x + S.pieces[q].y <= goal) q++;
        cta_piece[c] = std::min(q, np);
        S.cta_row[c] = c == 0 ? 0 : (q < np ? S.pieces[q].x : (int)N);
      }
      S.cta_row[0] = 0;
      cta_piece[0] = 0;
      for (int c = 1; c <= G; c++) {
        S.cta_row[c] = std::max(S.cta_row[c], S.cta_row[c - 1]);
        cta_piece[c] = std::max(cta_piece[c], cta_piece[c - 1]);
      }
      S.cta_row[G] = (int)N;
      cta_piece[G] = np;
      for (int c = 0; c < G; c++) {
        S.cta_tile[c] = (int)S.tiles.size();
        make_tiles(S.pieces, cta_piece[c], cta_piece[c + 1], S.tile_rows, S.tiles);
      }
      S.cta_tile[G] = (int)S.tiles.size();
    } else {
      const int64_t nw = tree ? S.tree.inst_win[1] : 0;
      for (int c = 0; c <= G; c++) {
        S.cta_row[c] = (int)(N * (int64_t)c / G);
        S.cta_win[c] = (int)(nw * c / G);
      }
    }
    S.grid_blocks = G;
  } else {
    S.order.resize(ni);
    for (int32_t i = 0; i < ni; i++) S.order[i] = i;
    std::stable_sort(S.order.begin(), S.order.end(),
                     [&](int a, int b) { return host.num_elem[a] > host.num_elem[b]; });
    // persistent CTAs: as many per SM as fit, or at most tile_ctas_per_sm (a tuned shape; results do
    // not depend on it)
    if (opt.tile_ctas_per_sm > 0) per_sm = std::min(per_sm, opt.tile_ctas_per_sm);
    S.grid_blocks = std::max(1, std::min<int>(dev_sms * std::max(per_sm, 1), ni));
    if (S.cluster) S.grid_blocks = ni * S.cluster;
    S.inst_tile.assign(ni + 1, 0);
    for (int32_t i = 0; segs && i < ni; i++) {
      S.inst_tile[i] = (int)S.tiles.size();
      make_tiles(S.pieces, inst_piece[i], inst_piece[i + 1], S.tile_rows, S.tiles);
    }
    S.inst_tile[ni] = (int)S.tiles.size();
  }
  S.tiles.push_back(np);  // sentinel: end piece of the last tile
  // device bytes, in the order implicit_init takes them
  const int m = opt.restart;
  size_t b = 0;
  b += al256(ld);                                           // rowf
  b += 5 * al256(8 * ld);                                   // cmdt, g64, wdx64, kdx64, inp64
  b += 2 * al256(8 * ld);                                   // diag, rhs
  b += al256(4 * ld) + al256(tb * ld);                      // gf, cdiag
  b += 2 * al256(tb * ld * (m + 1)) + al256(tb * ld);       // Wb, Z, y
  if (segs) b += 2 * al256(tb * ld);                        // pd, pc
  b += al256(sizeof(int2) * std::max<size_t>(1, S.pieces.size()));
  b += al256(4 * S.tiles.size());
  if (S.grid_mode)
    b += al256(4 * S.cta_row.size()) + al256(4 * S.cta_tile.size()) + al256(4 * S.cta_win.size());
  else
    b += al256(4 * S.inst_tile.size()) + al256(4 * S.order.size());
  b += 2 * al256(8 * S.inst_row.size()) + al256(4 * S.inst_n.size());
  b += al256(4) + al256(sizeof(double) * 2 * 4096 * kMaxDots);
  b += al256(sizeof(InstStat) * ni) + al256(sizeof(PackView)) + al256(sizeof(ImView));
  if (tree) {
    const TreePlan &T = S.tree;
    const size_t npc = std::max<size_t>(1, T.pmap.size());
    b += al256(ld) + al256(2 * T.wtp.size()) + al256(4 * T.wbase.size());
    b += al256(4 * npc) + al256(16 * npc) + al256(4 * std::max<size_t>(1, T.lev_off.size()));
    b += 3 * al256(4 * (size_t)(ni + 1));                   // inst_win, inst_piece, inst_lev
    b += 2 * al256(4 * tb * npc) + al256(8 * tb * npc) + al256(walk_bytes(tb, false) * npc);  // pmob, pstat, pval, gwalk
    b += al256(8 * npc) + al256(32 * npc);                  // pgf, pxb
    b += 4 * al256(tb * ld);                                // tinv, te, tbeta, talpha
    b += al256(4 * tb * T.wtp.size());                      // tent
  }
  bytes = b + 4096;
  return NRT_OK;
}

int Engine::implicit_init() {
  ImplicitState &S = *im;
  const int64_t N = host.ntot;
  const int32_t ni = host.ninst;
  const bool mixed = opt.precision == NRT_MIXED;
  const size_t tb = mixed ? 4 : 8;
  NRT_CUDA(cudaMemcpyAsync((void *)pv.topo, host.topo.data(), sizeof(Topo) * N,
                           cudaMemcpyHostToDevice, stream));
  cudaStream_t st = stream;
  ImView &iv = S.iv;
  const int64_t ld = (N + kRW - 1) & ~(int64_t)(kRW - 1);
  const bool tree = opt.precond == NRT_PRECOND_TREE, segs = opt.precond == NRT_PRECOND_SEGMENT;
  iv.ntot = N;
  iv.ld = ld;
  iv.win = S.win;
  iv.m = opt.restart;
  iv.precond = opt.precond;
  iv.krylov = opt.krylov;
  iv.scheme = opt.scheme;
  iv.tol_mode = opt.tol_mode;
  iv.tol = opt.tol;
  iv.max_iter = opt.max_iter;
  iv.inner_rel = !mixed ? 0.0 : (opt.inner_tol > 0 ? opt.inner_tol : NRT_INNER_TOL_DEFAULT);
  iv.rich = mixed && opt.precond == NRT_PRECOND_TREE && opt.krylov == NRT_GMRES &&
            opt.refinement == 0;
  iv.ninst = ni;
  iv.tile_rows = S.tile_rows;
  uint8_t *pr;
  TRYI(up(arena, pr, S.rowf.data(), N, st, ld)); iv.rowf = pr;
  // c_m dX / dT and the FP32 conductances are staged (filled in parallel, no zero fill
  // first); the other FP64 rows go up straight from the host pack
  std::unique_ptr<double[]> cmdt_b(new double[N]);
  std::unique_ptr<float[]> gf_b(new float[N]);
  double *cmdt = cmdt_b.get();
  float *gf = gf_b.get();
  parallel_ranges(N, [&](int64_t a, int64_t b) {
    for (int64_t j = a; j < b; j++) {
      cmdt[j] = host.c_m_dx[j] / host.inst[host.topo[j].flags >> INST_SHIFT].dT;
      gf[j] = (float)host.gax[j];
    }
  });
  double *p;
  TRYI(up(arena, p, cmdt, N, st, ld)); iv.cmdt = p;
  TRYI(up(arena, p, host.gax.data(), N, st, ld)); iv.g64 = p;
  TRYI(up(arena, p, host.wdx.data(), N, st, ld)); iv.wdx64 = p;
  TRYI(up(arena, p, host.kdx.data(), N, st, ld)); iv.kdx64 = p;
  TRYI(up(arena, p, host.inp.data(), N, st, ld)); iv.inp64 = p;
  TRYI(up(arena, iv.diag, (const double *)nullptr, ld, st));
  TRYI(up(arena, iv.rhs, (const double *)nullptr, ld, st));
  float *pf;
  TRYI(up(arena, pf, gf, N, st, ld)); iv.gf = pf;
  iv.cdiag = arena.take(tb * ld);
  if (!iv.cdiag) {
    set_error("arena exhausted");
    return NRT_ENOMEM;
  }
  const int m = opt.restart;
  iv.Wb = arena.take(tb * ld * (m + 1));
  iv.Z = arena.take(tb * ld * (m + 1));
  iv.yv = arena.take(tb * ld);
  iv.pcd = segs ? arena.take(tb * ld) : nullptr;
  iv.pcc = segs ? arena.take(tb * ld) : nullptr;
  if (!iv.Wb || !iv.Z || !iv.yv || (segs && (!iv.pcd || !iv.pcc))) {
    set_error("arena exhausted (Krylov workspace)");
    return NRT_ENOMEM;
  }
  NRT_CUDA(cudaMemsetAsync(iv.Wb, 0, tb * ld * (m + 1), st));
  NRT_CUDA(cudaMemsetAsync(iv.Z, 0, tb * ld * (m + 1), st));
  NRT_CUDA(cudaMemsetAsync(iv.yv, 0, tb * ld, st));
  int2 *pc;
  TRYI(up(arena, pc, S.pieces.data(), S.pieces.size(), st)); iv.pieces = pc;
  int *pi;
  TRYI(up(arena, pi, S.tiles.data(), S.tiles.size(), st)); iv.tiles = pi;
  if (S.grid_mode) {
    TRYI(up(arena, pi, S.cta_row.data(), S.cta_row.size(), st)); iv.cta_row = pi;
    TRYI(up(arena, pi, S.cta_tile.data(), S.cta_tile.size(), st)); iv.cta_tile = pi;
    TRYI(up(arena, pi, S.cta_win.data(), S.cta_win.size(), st)); iv.cta_win = pi;
  } else {
    TRYI(up(arena, pi, S.inst_tile.data(), S.inst_tile.size(), st)); iv.inst_tile = pi;
    TRYI(up(arena, pi, S.order.data(), S.order.size(), st)); iv.order = pi;
  }
  int64_t *pl;
  TRYI(up(arena, pl, S.inst_row.data(), S.inst_row.size(), st)); iv.inst_row = pl;
  TRYI(up(arena, pi, S.inst_n.data(), S.inst_n.size(), st)); iv.inst_n = pi;
  std::vector<int64_t> out(ni + 1, 0);
  for (int32_t i = 0; i < ni; i++) out[i + 1] = out[i] + host.num_elem[i];
  TRYI(up(arena, pl, out.data(), out.size(), st)); iv.inst_out = pl;
  TRYI(up(arena, iv.queue, (const int *)nullptr, 1, st));
  TRYI(up(arena, iv.partials, (const double *)nullptr, (size_t)2 * 4096 * kMaxDots, st));
  TRYI(up(arena, iv.stats, (const InstStat *)nullptr, ni, st));
  NRT_CUDA(cudaMemsetAsync(iv.stats, 0, sizeof(InstStat) * ni, st));
  if (tree) {
    const TreePlan &T = S.tree;
    const size_t npc = std::max<size_t>(1, T.pmap.size());
    uint8_t *p8;
    uint16_t *p16;
    int4 *p4;
    TRYI(up(arena, p8, T.pfl.data(), T.pfl.size(), st)); iv.pfl = p8;
    TRYI(up(arena, p16, T.wtp.data(), T.wtp.size(), st)); iv.wtp = p16;
    TRYI(up(arena, pi, T.wbase.data(), T.wbase.size(), st)); iv.wbase = pi;
    TRYI(up(arena, pi, T.pmap.data(), T.pmap.size(), st)); iv.pmap = pi;
    TRYI(up(arena, p4, T.plink.data(), T.plink.size(), st)); iv.plink = p4;
    TRYI(up(arena, pi, T.lev_off.data(), T.lev_off.size(), st)); iv.lev_off = pi;
    TRYI(up(arena, pi, T.inst_win.data(), T.inst_win.size(), st)); iv.inst_win = pi;
    TRYI(up(arena, pi, T.inst_piece.data(), T.inst_piece.size(), st)); iv.inst_piece = pi;
    TRYI(up(arena, pi, T.inst_lev.data(), T.inst_lev.size(), st)); iv.inst_lev = pi;
    iv.pmob = arena.take(4 * tb * npc);
    double *pd;
    TRYI(up(arena, pd, T.pgf.data(), T.pgf.size(), st)); iv.pgf = pd;
    iv.npieces = (int64_t)T.pmap.size();
    iv.pstat = arena.take(4 * tb * npc);
    iv.pval = arena.take(8 * tb * npc);
    iv.pxb = (double *)arena.take(32 * npc);
    iv.gwalk = arena.take(walk_bytes(tb, false) * npc);
    iv.tinv = arena.take(tb * ld);
    iv.te = arena.take(tb * ld);
    iv.tbeta = arena.take(tb * ld);
    iv.talpha = arena.take(tb * ld);
    iv.tent = arena.take(4 * tb * T.wtp.size());
    if (!iv.pmob || !iv.pstat || !iv.pval || !iv.pxb || !iv.gwalk || !iv.tinv || !iv.te || !iv.tbeta ||
        !iv.talpha || !iv.tent) {
      set_error("arena exhausted (tree preconditioner)");
      return NRT_ENOMEM;
    }
  }
  S.d_pv = (PackView *)arena.take(sizeof(PackView));
  S.d_iv = (ImView *)arena.take(sizeof(ImView));
  if (!S.d_pv || !S.d_iv) {
    set_error("arena exhausted (views)");
    return NRT_ENOMEM;
  }
  NRT_CUDA(cudaMemcpyAsync(S.d_pv, &pv, sizeof(PackView), cudaMemcpyHostToDevice, st));
  NRT_CUDA(cudaMemcpyAsync(S.d_iv, &iv, sizeof(ImView), cudaMemcpyHostToDevice, st));
  NRT_CUDA(cudaStreamSynchronize(st));
  return NRT_OK;
}

// Runs `nsteps` implicit steps for every instance (one launch).
static int implicit_launch(Engine &e, int nsteps, int force) {
  ImplicitState &S = *e.im;
  if (!S.grid_mode && !S.cluster) NRT_CUDA(cudaMemsetAsync(S.iv.queue, 0, sizeof(int), e.stream));
  const PackView *pv = S.d_pv;
  const ImView *iv = S.d_iv;
  double *V0 = e.V[0], *V1 = e.V[1];
  int cur = e.cur;
  // the drop-in per-call loop (force >= 0) has no device loop index: it is not recorded
  const RecView *rec = force < 0 ? e.record_view() : nullptr;
  void *args[] = {&pv, &iv, &nsteps, &force, &V0, &V1, &cur, &rec};
  if (S.grid_mode) {
    NRT_CUDA(cudaLaunchCooperativeKernel(S.kern, dim3(S.grid_blocks), dim3(kThreads), args, S.smem, e.stream));
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S.grid_blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = S.smem;
    cfg.stream = e.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)std::max(1, S.cluster);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = S.cluster ? 1 : 0;
    NRT_CUDA(cudaLaunchKernelExC(&cfg, S.kern, args));
  }
  count_launch_on(e.stream);
  return NRT_OK;
}

int Engine::implicit_step(int k, int force) {
  (void)k;
  return implicit_launch(*this, 1, force);
}

int implicit_advance(Engine &e, int64_t steps) {
  const int chunk = 64;
  while (steps > 0) {
    const int n = (int)std::min<int64_t>(chunk, steps);
    TRYI(implicit_launch(e, n, -1));
    TRYI(launch_advance_base(e.pv.inst, e.pv.ninst, n, e.stream));
    if (n & 1) e.cur ^= 1;
    e.steps_done += n;
    steps -= n;
  }
  return NRT_OK;
}

int instance_stats(Engine &e, int64_t *iters, int32_t *last_iters, int32_t *nonconv,
                   double *last_res) {
  const int32_t ni = e.host.ninst;
  std::vector<InstStat> s(ni, InstStat{0, 0, 0, 0.0, 0, 0, 0, 0, 0});
  if (e.im) {
    NRT_CUDA(cudaMemcpyAsync(s.data(), e.im->iv.stats, sizeof(InstStat) * ni,
                             cudaMemcpyDeviceToHost, e.stream));
    NRT_CUDA(cudaStreamSynchronize(e.stream));
  }
  for (int32_t i = 0; i < ni; i++) {
    if (iters) iters[i] = s[i].iters;
    if (last_iters) last_iters[i] = s[i].last_iters;
    if (nonconv) nonconv[i] = s[i].nonconv;
    if (last_res) last_res[i] = s[i].last_res;
  }
  return NRT_OK;
}

int pass_counts(Engine &e, int64_t *residuals, int64_t *applies, int64_t *xupdates,
                int64_t *basis, int64_t *rich) {
  const int32_t ni = e.host.ninst;
  std::vector<InstStat> s(ni, InstStat{0, 0, 0, 0.0, 0, 0, 0, 0, 0});
  if (e.im) {
    NRT_CUDA(cudaMemcpyAsync(s.data(), e.im->iv.stats, sizeof(InstStat) * ni,
                             cudaMemcpyDeviceToHost, e.stream));
    NRT_CUDA(cudaStreamSynchronize(e.stream));
  }
  for (int32_t i = 0; i < ni; i++) {
    if (residuals) residuals[i] = s[i].residuals;
    if (applies) applies[i] = s[i].applies;
    if (xupdates) xupdates[i] = s[i].xupdates;
    if (basis) basis[i] = s[i].basis;
    if (rich) rich[i] = s[i].rich;
  }
  return NRT_OK;
}

// NRT_EDEVICE when a bounded wait of an explicit kernel gave up (the pack's error word is set; the
// implicit kernels wait for nothing but their own CTAs); synchronises.
int device_check(Engine &e) {
  int err = 0;
  if (e.pv.err && e.opt.mode == NRT_EXPLICIT)
    NRT_CUDA(cudaMemcpyAsync(&err, e.pv.err, sizeof(int), cudaMemcpyDeviceToHost, e.stream));
  NRT_CUDA(cudaStreamSynchronize(e.stream));
  if (err) {
    set_error("explicit step: a bounded wait for its tile copies expired");
    return NRT_EDEVICE;
  }
  return NRT_OK;
}

__global__ void compact_rows(const double *__restrict__ V, double *__restrict__ out,
                             const int64_t *__restrict__ from, const int *__restrict__ n,
                             const int64_t *__restrict__ to) {
  const int i = blockIdx.x;
  const double *src = V + from[i];
  double *dst = out + to[i];
  for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < n[i]; j += gridDim.y * blockDim.x) dst[j] = src[j];
}

// The Krylov workspace, dead between steps, takes the packed copy: Wb holds m + 1 >= 2 rows
// of at least 4 bytes each.
int implicit_compact(Engine &e, const double *&src, int64_t &n) {
  const int32_t ni = e.host.ninst;
  int64_t total = 0;
  for (int32_t i = 0; i < ni; i++) total += e.host.num_elem[i];
  n = total;
  if (total == e.host.ntot) return NRT_OK;  // no padding
  ImplicitState &S = *e.im;
  double *out = (double *)S.iv.Wb;
  // as many CTAs per instance as leave each a few rows per thread (two trees of 100,000: the whole
  // call 111 us with one CTA each, 25 so)
  const int largest = *std::max_element(e.host.num_elem.begin(), e.host.num_elem.end());
  const dim3 grid(ni, std::max(1, std::min(64, largest / 2048)));
  compact_rows<<<grid, 256, 0, e.stream>>>(src, out, S.iv.inst_row, S.iv.inst_n, S.iv.inst_out);
  count_launch_on(e.stream);
  NRT_CUDA(cudaGetLastError());
  src = out;
  return NRT_OK;
}

// Sum of non-converged steps over all instances (-1 on a CUDA error); waits for the stream.
int64_t nonconverged_total(Engine &e) {
  if (!e.im) return 0;
  std::vector<InstStat> s(e.host.ninst);
  if (cudaMemcpyAsync(s.data(), e.im->iv.stats, sizeof(InstStat) * s.size(), cudaMemcpyDeviceToHost,
                      e.stream) != cudaSuccess ||
      cudaStreamSynchronize(e.stream) != cudaSuccess)
    return -1;
  int64_t t = 0;
  for (const InstStat &x : s) t += x.nonconv;
  e.nonconv_seen = t;
  return t;
}

void Engine::implicit_release() {
  delete im;
  im = nullptr;
}

int Engine::get_stats(nrt_stats *st) {
  memset(st, 0, sizeof(*st));
  st->steps = steps_done;
  st->device_bytes = (int64_t)device_bytes();
  if (opt.mode == NRT_IMPLICIT_BE && im) {
    std::vector<InstStat> s(host.ninst);
    NRT_CUDA(cudaMemcpyAsync(s.data(), im->iv.stats, sizeof(InstStat) * host.ninst,
                             cudaMemcpyDeviceToHost, stream));
    NRT_CUDA(cudaStreamSynchronize(stream));
    for (const InstStat &x : s) {
      st->krylov_iters += x.iters;
      st->nonconverged_steps += x.nonconv;
      st->last_iters = std::max(st->last_iters, x.last_iters);
      st->last_residual = std::max(st->last_residual, x.last_res);
    }
  }
  return NRT_OK;
}

// Expands the stored symmetric system to the reference's CSR (src/solverIm-cpu.cpp:29-183
// column order: mother, diagonal, DR, DL; identity rows 1).  Runs an assembly-only pass
// for the next step and restores the state it touched.
int export_system(Engine &e, int input_active, int32_t *row_ptr, int32_t *col, double *val,
                  double *rhs, int32_t *nnz_out) {
  if (e.opt.mode != NRT_IMPLICIT_BE || e.host.ninst != 1) {
    set_error("export_system needs a single-tree implicit solver");
    return NRT_EINVAL;
  }
  const int64_t N = e.host.ntot;
  const bool mixed = e.opt.precision == NRT_MIXED;
  const size_t gb = (mixed ? 4 : 8) * 3 * N;
  void *gate = mixed ? (void *)e.pv.gatef : (void *)e.pv.gate;
  std::vector<char> saved(gb);
  std::vector<double> Vother(N);
  ImplicitState &S = *e.im;
  InstStat stat0;
  NRT_CUDA(cudaMemcpyAsync(saved.data(), gate, gb, cudaMemcpyDeviceToHost, e.stream));
  NRT_CUDA(cudaMemcpyAsync(Vother.data(), e.V[e.cur ^ 1], 8 * N, cudaMemcpyDeviceToHost, e.stream));
  NRT_CUDA(cudaMemcpyAsync(&stat0, S.iv.stats, sizeof(InstStat), cudaMemcpyDeviceToHost, e.stream));
  NRT_CUDA(cudaStreamSynchronize(e.stream));
  const int saved_iter = S.iv.max_iter;
  S.iv.max_iter = -1;  // assembly only
  NRT_CUDA(cudaMemcpyAsync(S.d_iv, &S.iv, sizeof(ImView), cudaMemcpyHostToDevice, e.stream));
  int rc = implicit_launch(e, 1, input_active ? 1 : 0);
  S.iv.max_iter = saved_iter;
  const cudaError_t ce = cudaMemcpyAsync(S.d_iv, &S.iv, sizeof(ImView), cudaMemcpyHostToDevice, e.stream);
  if (rc) return rc;
  NRT_CUDA(ce);
  std::vector<double> diag(N), rh(N), g(N);
  NRT_CUDA(cudaMemcpyAsync(diag.data(), S.iv.diag, 8 * N, cudaMemcpyDeviceToHost, e.stream));
  NRT_CUDA(cudaMemcpyAsync(rh.data(), S.iv.rhs, 8 * N, cudaMemcpyDeviceToHost, e.stream));
  NRT_CUDA(cudaMemcpyAsync(g.data(), S.iv.g64, 8 * N, cudaMemcpyDeviceToHost, e.stream));
  NRT_CUDA(cudaMemcpyAsync(gate, saved.data(), gb, cudaMemcpyHostToDevice, e.stream));
  NRT_CUDA(cudaMemcpyAsync(e.V[e.cur ^ 1], Vother.data(), 8 * N, cudaMemcpyHostToDevice, e.stream));
  NRT_CUDA(cudaMemcpyAsync(S.iv.stats, &stat0, sizeof(InstStat), cudaMemcpyHostToDevice, e.stream));
  NRT_CUDA(cudaStreamSynchronize(e.stream));
  int32_t nnz = 0;
  const int64_t n = e.host.num_elem[0];  // without the padding
  for (int64_t j = 0; j < n; j++) {
    const Topo &t = e.host.topo[j];
    row_ptr[j] = nnz;
    if (t.flags & F_IDENT) {
      col[nnz] = (int32_t)j;
      val[nnz++] = 1.0;
      rhs[j] = Vother[j];
      continue;
    }
    if (t.flags & F_UP) { col[nnz] = t.mother; val[nnz++] = -g[j]; }
    col[nnz] = (int32_t)j;
    val[nnz++] = diag[j];
    if (t.flags & F_DOWNR) { col[nnz] = (int32_t)j + 1; val[nnz++] = -g[j + 1]; }
    if (t.flags & F_DOWNL) { col[nnz] = t.dl; val[nnz++] = -g[t.dl]; }
    rhs[j] = rh[j];
  }
  row_ptr[n] = nnz;
  *nnz_out = nnz;
  return NRT_OK;
}

}  // namespace nrt
