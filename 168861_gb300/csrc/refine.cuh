// Mixed-precision step with the tree preconditioner, by windows (included by implicit.cu).
//
// The step's passes over the rows are fused to four:
//   - refine_assemble: gates, W, K, diagonal, right-hand side, the first residual (a row per
//     thread), and the pieces' matrices of the factorisation (four rows per thread, as in the
//     passes below);
//   - tree_pivots (tree.cuh): the factorisation and the elimination of that residual;
//   - refine_update<true>: substitution, x += z, the FP64 residual of the new x, and its
//     elimination, for the next refinement cycle;
//   - refine_update<false>: the same without the elimination (from the second cycle on, which
//     is nearly always the last).
// Between them one CTA walks the pieces.  The walk also forms the new potential of every
// piece's first and last row, so that a window needs nothing of another one's new potential
// from the pass that is writing it; those rows take the walk's value, bit for bit what their
// neighbours' residuals use.  Against separate passes (assembly, matrices, pivots, and per
// cycle elimination, substitution, update, residual) a row-step moves about 230 bytes
// instead of 300 and needs six fewer passes' latencies and, on the one-tree launch, 4 syncs
// of the grid instead of 14.
#pragma once

namespace nrt {

// x of the row before this thread's first and after its last, in the window.  ends: 2 * kWarps
// doubles; one CTA barrier.
__device__ __forceinline__ void window_ends(const double (&x)[kRW], double *ends, double &xm,
                                            double &xp) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  xm = __shfl_up_sync(0xffffffffu, x[kRW - 1], 1);
  xp = __shfl_down_sync(0xffffffffu, x[0], 1);
  if (lane == 31) ends[w] = x[kRW - 1];
  if (lane == 0) ends[kWarps + w] = x[0];
  __syncthreads();
  if (lane == 0 && w > 0) xm = ends[w - 1];
  if (lane == 31 && w + 1 < kWarps) xp = ends[kWarps + w + 1];
}

// The sums of a pass (||b||^2, ||r||^2) are taken by chunks of whole windows, up to kSumChunks of
// them, whose edges depend on the tree alone: as with rows_reduce, the result does not depend on how
// many CTAs share the tree, and so not on the trees beside it.  After a chunk a warp leaves kG numbers
// in S.wpart (of two sums four each) and starts afresh, and after the pass a warp sums each chunk's.
// Against one sum per CTA, whose bits changed with the cluster's size, clusters take the same time and
// batches of one CTA per tree 2 to 5 % more (8 steps of 1000 trees of 1e3 to 3e4: 9.5 -> 9.8 ms, 320
// of them 7.8 -> 8.2, the 2048 trees of 1e3 to 1e5 36.3 -> 37.1).  Forms measured and not taken: the
// passes called once per chunk (37.5 for the last), every chunk summed up where it ends (37.6), every
// thread's parts in shared memory (37.2 with 24 KB of it, 1000 trees 10.4).
template <int kN>
__device__ __forceinline__ void leave_chunk(const Shared &S, int chunk, double a, double b) {
  static_assert(kG == 8 && kWarps == 8, "a warp's places in S.wpart");
  const int lane = threadIdx.x & 31;
  double *to = S.wpart + (chunk * kWarps + (threadIdx.x >> 5)) * kG;
#pragma unroll
  for (int o = 16; o >= (kN == 1 ? 8 : 4); o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    if (kN == 2) b += __shfl_down_sync(0xffffffffu, b, o);
  }
  if (lane < kG / kN) {
    to[lane] = a;
    if (kN == 2) to[lane + kG / 2] = b;
  }
}

// kN sums to S.red[0 ..].
template <int kMode, int kN>
__device__ __forceinline__ void sum_windows(const Ctx<float, kMode> &c, Shared &S, double *partials,
                                            int &parity) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  double *sum = chunk_sums<kMode>(S, partials, parity);
  for (int v = w; v < c.wv1 - c.wv0; v += kWarps) {
    const double *from = S.wpart + v * kWarps * kG + lane;
    double x = 0;
    if (kMode != kGrid || c.w0 < c.w1) x = from[0] + from[32];  // lane & 7: the place of a warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (kN == 1 || o != 4) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0 || (kN == 2 && lane == 4)) sum[(c.wv0 + v) * kMaxDots + (lane >> 2)] = x;
  }
  total_chunks<kMode>(kN, c.wchunks, sum, S, partials, parity, 0);
}

// kCn: Crank-Nicolson.  The rows' part takes one row per thread, a warp 32 neighbours: with the
// four rows per thread that the matrices' scan wants, its loads used half of each sector and its
// numbers did not fit the registers (22 accesses of local memory per row and step, most of them
// L2 round trips).  2048 trees of 1e3 to 1e5: 39.2 -> 38.2 ms for 8 steps; one tree of 30k, whose
// windows are smaller than a CTA's threads times four: 3.35 -> 3.13 ms for 32.
// What is left is bound by the FP64 pipe's latency and rate (16 cycles of an SM per warp's
// operation), so rare rows share one x0 with the warp's ends, and x0 goes to Z for the passes that
// would form it again (the pieces' ends, the first update): 3.13 -> 3.00 ms, 38.2 -> 37.8 ms.
template <int kMode, bool kCn>
__device__ __noinline__ void refine_assemble(const Ctx<float, kMode> &c, const double *Vin,
                                             const double *Vout, int active, int inst) {
  const PackView &pv = *c.pv;
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const int64_t N = pv.ntot;
  float *gate = pv.gatef;
  const bool dense = pv.hh_dense != 0;
  const int lane = threadIdx.x & 31;
  float bacc = 0;
  double racc = 0;
  int chunk = 0;
  for (int w = c.w0; w < c.w1; w++) {
    const int64_t r0 = c.wrow0 + (int64_t)(w - c.iw0) * iv.win;
    const int nr = (int)min((int64_t)iv.win, c.wend - r0);
#pragma unroll 1
    for (int l = threadIdx.x; l - lane < nr; l += kThreads) {
      const int64_t row = min(r0 + l, N - 1);
      const bool ok = l < nr;
      const double v = Vin[row], o = Vout[row], cm = iv.cmdt[row], g = iv.g64[row];
      const uint32_t f = ok ? iv.rowf[row] : R_IDENT;
      float gm = 0, gh = 0, gn = 0;
      if (dense || (f & R_HH)) {
        gm = gate[row];
        gh = gate[N + row];
        gn = gate[2 * N + row];
      }
      const double x = 2.0 * v - o;
      double xm = __shfl_up_sync(0xffffffffu, x, 1), xp = __shfl_down_sync(0xffffffffu, x, 1);
      double gdn = __shfl_down_sync(0xffffffffu, g, 1), vm = 0, vp = 0;
      if (kCn) {
        vm = __shfl_up_sync(0xffffffffu, v, 1);
        vp = __shfl_down_sync(0xffffffffu, v, 1);
      }
      if (!ok) continue;  // the loop's bound is the warp's
      double wdx = 0.0, kdx = 0.0;
      if (f & R_HH) {  // identity rows' gates move too
        const HHParams32 q = hh_params32(
            pv.hpq, pv.hp_cls ? (int64_t)pv.hp_cls[row] : (pv.hp_inst ? (int64_t)inst : row));
        const float dv = d2f(v - f2d(q.v[HP_REST]));
        const GateStep32 s = hh_step32(dv + q.v[HP_LSNA], dv + q.v[HP_LSK], gm, gh, gn, q.v[HP_DTMS],
                                       q.v[HP_GNA], q.v[HP_GK], q.v[HP_GL], q.v[HP_ENA], q.v[HP_EK],
                                       q.v[HP_EL]);
        gate[row] = s.m;
        gate[N + row] = s.h;
        gate[2 * N + row] = s.n;
        wdx = f2d(s.W * q.v[HP_DX]);
        kdx = f2d(s.K * q.v[HP_DX]);
      } else if (!(f & R_IDENT)) {
        wdx = iv.wdx64[row];
        kdx = iv.kdx64[row];
      }
      // the neighbour that is not in the warp (the rows before and after it, a DL child, a far
      // mother): one for nearly every row that has any, so one x0 for all of the warp
      const bool dl = f & R_DOWNL, far = f & R_FAR, rare = dl || far;
      double gl = 0.0, xl = 0.0, vl = 0.0;
      if (rare || lane == 0 || lane == 31) {
        int tm = 0, tl = 0;
        if (rare) {
          const Topo t = pv.topo[row];
          tm = t.mother;
          tl = t.dl;
        }
        const int64_t qm = far ? (int64_t)tm : max(row - 1, (int64_t)0), qp = min(row + 1, N - 1);
        const int64_t q = dl ? (int64_t)tl : (far || lane == 0) ? qm : qp;
        const double ev = Vin[q], ex = 2.0 * ev - Vout[q], eg = iv.g64[q];
        if (dl) {
          gl = eg;
          xl = ex;
          vl = ev;
        } else if (far || lane == 0) {
          xm = ex;
          vm = ev;
        } else {
          xp = ex;
          vp = ev;
          gdn = eg;
        }
        if (dl && (far || lane == 0)) {
          xm = x0_of(Vin, Vout, qm);
          if (kCn) vm = Vin[qm];
        }
        if (rare && lane == 31) {
          xp = x0_of(Vin, Vout, qp);
          if (kCn) vp = Vin[qp];
          gdn = iv.g64[qp];
        }
      }
      // columns that are not there: nothing of another tree's rows gets in
      double gup = g;
      if (!(f & R_UP)) gup = xm = vm = 0.0;
      if (!(f & R_DOWNR)) gdn = xp = vp = 0.0;
      const double cj = (kCn ? 2.0 * cm : cm) - wdx;
      double d = (cj + gdn) + gup, b;
      if (!kCn) {
        b = fma(cm, v, kdx);
      } else {  // (2 c_m dX/dT + W dX) V^n - sum g (V^n - V^n_q) + 2 (K dX + I)
        b = (2.0 * cm + wdx) * v;
        b -= gup * (v - vm);
        b -= gdn * (v - vp);
        b += 2.0 * kdx;
      }
      if (dl) {
        d += gl;
        if (kCn) b -= gl * (v - vl);
      }
      if (active && (f & R_INP)) b += kCn ? 2.0 * iv.inp64[row] : iv.inp64[row];
      double res = fma(-d, x, b);
      res = fma(gup, xm, res);
      res = fma(gdn, xp, res);
      if (dl) res = fma(gl, xl, res);
      if (f & R_IDENT) b = res = 0.0;
      x0_store(c.w.Z, iv.ld, row, (f & R_IDENT) ? o : x);
      iv.diag[row] = d;
      iv.rhs[row] = b;
      ((float *)iv.cdiag)[row] = d2f(cj);
      c.w.Wb[row] = d2f(res);
      const float bf = d2f(b);
      bacc += bf * bf;
      racc += res * res;
    }
    __syncthreads();  // the window's rows are there
    WinRows<float, kMode> r(c, iv, w);
    float cc[kRW] = {}, gf[kRW] = {};
    if (r.ok) {
      ld_rows((const float *)iv.cdiag + r.rb, cc);
      ld_rows((const float *)iv.gf + r.rb, gf);
    }
    r.ids(c, iv);
    window_maps(r, cc, gf, (Mob<float> *)iv.pmob + c.ip0,
                (float *)iv.tent + 4 * thread_slot(iv, w), (float *)S.warp);
    if (w + 1 == c.wend_of[chunk]) {
      leave_chunk<2>(S, chunk, f2d(bacc), racc);
      bacc = 0;
      racc = 0;
      chunk++;
    }
  }
}

struct RefineX {
  float4 s, v;  // pstat, pval
  double2 b;    // the potential of the piece's first and last row before the update
};

// The walks of one refinement cycle, with the new potential of the pieces' first and last
// rows (in a group: of this CTA's pieces and the ones next to them).  pb: the buffer of the
// pieces' values.
template <int kMode>
__device__ __noinline__ void refine_walk(const Ctx<float, kMode> &c, int pb) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<float> k = walk_of(c, iv, S);
  const float4 *ps = (const float4 *)iv.pstat + c.ip0;
  const float4 *pa = (const float4 *)iv.pval + (c.ip0 + (int64_t)pb * iv.npieces);
  const double2 *px = (const double2 *)iv.pxb + (c.ip0 + (int64_t)pb * iv.npieces);
  const int4 *lk = iv.plink + c.ip0;
  auto up = [](const Mob<float> &x, float s) { return x.c + x.a * s; };
  auto last = [](float B, float bL, float aL, float y, float zp) { return aL + bL * y + B * zp; };
  auto put = [&](int q, const RefineX &x, float y, float zp, float zl, bool one) {
    const float zf = x.v.z + x.s.z * y + x.s.w * zp;
    const double xl = x.b.y + f2d(zl);
    k.px[q] = make_double2(one ? xl : x.b.x + f2d(zf), xl);  // one row: first is last
  };
  auto get = [&](int q) {
    const float4 a = ps[q], b = pa[q];
    return Mob<float>{a.x, a.y, b.x, b.y};
  };
  if (staged(c, iv)) {
#pragma unroll 4
    for (int q = threadIdx.x; q < c.np; q += kThreads) k.st[q] = get(q);
    __syncthreads();
    auto sget = [&](int q) { return k.st[q]; };
    walk_up<float, kMode, Mob<float>>(c, iv, k, sget, up);
    walk_down<float, kMode, Mob<float>>(c, iv, k, sget,
                                        [&](int, const Mob<float> &x, float y, float zp) {
                                          return last(x.a, x.b, x.d, y, zp);
                                        });
    auto one = [&](int q) {
      if (q == kNoPiece) return;
      put(q, RefineX{ps[q], pa[q], px[q]}, k.yin[q], k.zpar[q], k.val[q], k.link[q].w != 0);
    };
    if (one_cta(kMode)) {
      for (int q = threadIdx.x; q < c.np; q += kThreads) one(q);
      __syncthreads();
      return;
    }
    const int a = c.w0 < c.w1 ? iv.wbase[c.w0] : 0;
    const int b = c.w0 < c.w1 ? (c.w1 < c.iw1 ? iv.wbase[c.w1] : c.np) : 0;
    for (int o = a + threadIdx.x; o < b; o += kThreads) {
      const int q = iv.pmap[c.ip0 + o];
      const ushort4 t = k.link[q];
      one(q);
      one(t.x);
      one(t.y);
      one(t.z);
    }
    __syncthreads();
    return;
  }
  walk_up<float, kMode, Mob<float>>(c, iv, k, get, up);
  auto getx = [&](int q) { return RefineX{ps[q], pa[q], px[q]}; };
  walk_down<float, kMode, RefineX>(c, iv, k, getx, [&](int q, const RefineX &x, float y, float zp) {
    const float zl = last(x.s.x, x.s.y, x.v.y, y, zp);
    put(q, x, y, zp, zl, lk[q].w != 0);
    return zl;
  });
}

// x += z by substitution, then the FP64 residual b - A x; leaves the warps' parts of
// ||scale r||^2, of FP32 sums per thread (see ph_residual).  kElim, the step's first cycle: x starts from the
// initial guess, and r is eliminated into buffer pb of the pieces' values; else x is updated in
// Vout and r stored (W_0).
template <int kMode, bool kElim>
__device__ __noinline__ void refine_update(const Ctx<float, kMode> &c, double *Vout, float scale, int pb) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<float> k = walk_of(c, iv, S);
  float *scz = (float *)S.warp, *sc0 = scz + 2 * kWarps, *sc1 = sc0 + 2 * kWarps;
  double *ends = S.warp + 4 * kWarps;
  float *pval = (float *)iv.pval + 4 * ((int64_t)c.ip0 + (int64_t)pb * iv.npieces);
  double *pxb = (double *)iv.pxb + 2 * ((int64_t)c.ip0 + (int64_t)pb * iv.npieces);
  float acc = 0;
  int chunk = 0;
  for (int w = c.w0; w < c.w1; w++) {
    WinRows<float, kMode> r(c, iv, w);
    const int64_t rb = r.rb;
    float al[kRW] = {}, ee[kRW] = {}, inv[kRW] = {}, be[kRW] = {};
    double x[kRW] = {};
    if (r.ok) {
      ld_rows((const float *)iv.talpha + rb, al);
      ld_rows((const float *)iv.te + rb, ee);
      ld_rows((const float *)iv.tinv + rb, inv);
      ld_rows((const float *)iv.tbeta + rb, be);
      if (kElim) x0_rows(c.w.Z, iv.ld, rb, x);
      else ld_rows(Vout + rb, x);
    }
    r.ids(c, iv);
    // substitution
    float A[1] = {0}, M = 1, y[1];
#pragma unroll
    for (int u = 0; u < kRW; u++) {
      if (r.is(u, P_IDENT)) continue;
      al[u] = inv[u] * (al[u] + be[u] * k.yin[r.pid[u]]);
      if (r.is(u, P_FIRST)) {
        al[u] += ee[u] * k.zpar[r.pid[u]];
        A[0] = al[u];
        M = 0;
      } else {
        A[0] = al[u] + ee[u] * A[0];
        M *= ee[u];
      }
    }
    affine_enter<float, 1, false>(A, M, scz, y, r.idle, false);
    float cur = y[0];
#pragma unroll
    for (int u = 0; u < kRW; u++) {
      if (r.is(u, P_IDENT)) continue;
      if (!r.is(u, P_FIRST)) al[u] += ee[u] * cur;
      cur = al[u];
      x[u] += f2d(cur);
      if (r.is(u, P_FIRST)) x[u] = k.px[r.pid[u]].x;
      if (r.is(u, P_LAST)) x[u] = k.px[r.pid[u]].y;
    }
    if (r.ok) st_rows(Vout + rb, x);
    double xm, xp;
    window_ends(x, ends, xm, xp);
    // residual
    double rh[kRW] = {}, dg[kRW] = {}, g[kRW] = {}, gnext = 0;
    if (r.ok) {
      ld_rows((const double *)iv.rhs + rb, rh);
      ld_rows((const double *)iv.diag + rb, dg);
      ld_rows(iv.g64 + rb, g);
      gnext = iv.g64[rb + kRW < iv.ld ? rb + kRW : iv.ld - 1];
    }
#pragma unroll
    for (int u = 0; u < kRW; u++) {
      if (r.is(u, P_IDENT)) {
        al[u] = 0;
        continue;
      }
      double mo = u > 0 ? x[u > 0 ? u - 1 : 0] : xm;
      double nx = u + 1 < kRW ? x[u + 1 < kRW ? u + 1 : 0] : xp, gl = 0, xl = 0;
      if (r.is(u, P_FIRST | P_LAST)) {
        const int4 lk = iv.plink[c.ip0 + r.pid[u]];
        if (r.is(u, P_FIRST) && lk.z >= 0) mo = k.px[lk.z].y;
        if (r.is(u, P_LAST)) {
          if (lk.x >= 0) nx = k.px[lk.x].x;
          if (r.is(u, R_DOWNL)) {
            gl = iv.pgf[c.ip0 + lk.y];
            xl = k.px[lk.y].x;
          }
        }
      }
      double s = fma(-dg[u], x[u], rh[u]);
      if (r.is(u, P_UP)) s = fma(g[u], mo, s);
      if (r.is(u, R_DOWNR)) s = fma(u + 1 < kRW ? g[u + 1 < kRW ? u + 1 : 0] : gnext, nx, s);
      if (r.is(u, R_DOWNL)) s = fma(gl, xl, s);
      al[u] = d2f(s);
      const float e = al[u] * scale;
      acc = fmaf(e, e, acc);
    }
    if (kElim) {
#pragma unroll
      for (int u = 0; u < kRW; u++) {
        if (r.is(u, P_FIRST)) pxb[2 * (int64_t)r.pid[u]] = x[u];
        if (r.is(u, P_LAST)) pxb[2 * (int64_t)r.pid[u] + 1] = x[u];
      }
      window_eliminate(r, al, ee, inv, be, pval, sc0, sc1);
      if (r.ok) st_rows((float *)iv.talpha + rb, al);
    } else if (r.ok) {
      st_rows(c.w.Wb + rb, al);
    }
    if (w + 1 == c.wend_of[chunk]) {
      leave_chunk<1>(S, chunk, f2d(acc), 0.0);
      acc = 0;
      chunk++;
    }
  }
}

}  // namespace nrt
