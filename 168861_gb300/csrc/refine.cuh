// Mixed-precision step with the tree preconditioner, by windows (included by implicit.cu).
//
// The step's passes over the rows are fused to four, each reading its rows in row order with
// 16-byte loads, four rows per thread:
//   - refine_assemble: gates, W, K, diagonal, right-hand side, the first residual, and the
//     pieces' matrices of the factorisation;
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
  if (lane == 31) ends[w] = x[kRW - 1];
  if (lane == 0) ends[kWarps + w] = x[0];
  __syncthreads();
  xm = __shfl_up_sync(0xffffffffu, x[kRW - 1], 1);
  xp = __shfl_down_sync(0xffffffffu, x[0], 1);
  if (lane == 0 && w > 0) xm = ends[w - 1];
  if (lane == 31 && w + 1 < kWarps) xp = ends[kWarps + w + 1];
}

// kCn: Crank-Nicolson.
template <int kMode, bool kCn>
__device__ __noinline__ double2 refine_assemble(Ctx<float, kMode> c, const double *Vin,
                                                const double *Vout, int active, int inst) {
  const PackView &pv = *c.pv;
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const int64_t N = pv.ntot;
  float *gate = pv.gatef;
  const bool dense = pv.hh_dense != 0;
  float bacc = 0;
  double racc = 0;
  int par = 0;
  for (int w = c.w0; w < c.w1; w++) {
    float *sc = (float *)S.warp + par * 5 * kWarps;
    par ^= 1;
    WinRows<float, kMode> r(c, iv, w);
    const int64_t rb = r.rb;
    float cc[kRW] = {}, gf[kRW] = {}, rr4[kRW] = {};
    if (r.ok) {
      double v[kRW], xv[kRW], cm[kRW], g[kRW];
      ld_rows(Vin + rb, v);
      ld_rows(Vout + rb, xv);
      ld_rows(iv.cmdt + rb, cm);
      ld_rows(iv.g64 + rb, g);
      const int64_t rm = rb > 0 ? rb - 1 : 0, rp = rb + kRW < N ? rb + kRW : N - 1;
      const double vmo = Vin[rm], vno = Vin[rp], omo = Vout[rm], ono = Vout[rp];
      const double gnext = iv.g64[rp];
      const uint32_t rf = *(const uint32_t *)(iv.rowf + rb);
      float g0[kRW] = {}, g1[kRW] = {}, g2[kRW] = {};
      if (dense) {
        ld_rows(gate + rb, g0);
        ld_rows(gate + N + rb, g1);
        ld_rows(gate + 2 * N + rb, g2);
      }
      uint4 cls = make_uint4(0, 0, 0, 0);
      if (pv.hp_cls) cls = *(const uint4 *)(pv.hp_cls + rb);
      const double xm = 2.0 * vmo - omo, xp = 2.0 * vno - ono;
#pragma unroll
      for (int u = 0; u < kRW; u++) xv[u] = 2.0 * v[u] - xv[u];  // x0
      double dg[kRW], rh[kRW];
#pragma unroll
      for (int u = 0; u < kRW; u++) {
        const int64_t row = rb + u;
        const uint32_t f = (rf >> (8 * u)) & 0xffu;
        dg[u] = rh[u] = 0.0;
        float wdxf, kdxf;
        double wdx, kdx;
        if (!r.is(u, P_IDENT) || (f & R_HH)) {  // identity rows' gates move too
          if (f & R_HH) {
            if (!dense) {
              g0[u] = gate[row];
              g1[u] = gate[N + row];
              g2[u] = gate[2 * N + row];
            }
            const uint32_t cl = u == 0 ? cls.x : u == 1 ? cls.y : u == 2 ? cls.z : cls.w;
            const HHParams32 q =
                hh_params32(pv.hpq, pv.hp_cls ? (int64_t)cl : (pv.hp_inst ? (int64_t)inst : row));
            const float dv = d2f(v[u] - f2d(q.v[HP_REST]));
            GateStep32 s = hh_step32(dv + q.v[HP_LSNA], dv + q.v[HP_LSK], g0[u], g1[u], g2[u],
                                     q.v[HP_DTMS], q.v[HP_GNA], q.v[HP_GK], q.v[HP_GL],
                                     q.v[HP_ENA], q.v[HP_EK], q.v[HP_EL]);
            g0[u] = s.m;
            g1[u] = s.h;
            g2[u] = s.n;
            if (!dense) {
              gate[row] = s.m;
              gate[N + row] = s.h;
              gate[2 * N + row] = s.n;
            }
            wdxf = s.W * q.v[HP_DX];
            kdxf = s.K * q.v[HP_DX];
            wdx = f2d(wdxf);
            kdx = f2d(kdxf);
          } else {
            wdx = iv.wdx64[row];
            kdx = iv.kdx64[row];
          }
        }
        if (r.is(u, P_IDENT)) continue;
        const double gn = u + 1 < kRW ? g[u + 1 < kRW ? u + 1 : 0] : gnext;
        const double cj = (kCn ? 2.0 * cm[u] : cm[u]) - wdx;
        double d = cj, gl = 0.0, xl = 0.0, xmo = u > 0 ? xv[u > 0 ? u - 1 : 0] : xm;
        double vmother = u > 0 ? v[u > 0 ? u - 1 : 0] : vmo, vl = 0.0;
        if (f & (R_DOWNL | R_FAR)) {
          const Topo t = pv.topo[row];
          if (f & R_DOWNL) {
            gl = iv.g64[t.dl];
            xl = x0_of(Vin, Vout, t.dl);
            if (kCn) vl = Vin[t.dl];
            d += gl;
          }
          if (f & R_FAR) {
            xmo = x0_of(Vin, Vout, t.mother);
            vmother = Vin[t.mother];
          }
        }
        if (f & R_DOWNR) d += gn;
        if (f & R_UP) d += g[u];
        dg[u] = d;
        cc[u] = d2f(cj);
        if (f & R_UP) gf[u] = d2f(g[u]);
        const bool inj = active && (f & R_INP);
        double b;
        if (!kCn) {
          b = cm[u] * v[u] + kdx;
          if (inj) b += iv.inp64[row];
        } else {  // (2 c_m dX/dT + W dX) V^n - sum g (V^n - V^n_q) + 2 (K dX + I)
          b = (2.0 * cm[u] + wdx) * v[u];
          if (f & R_UP) b -= g[u] * (v[u] - vmother);
          if (f & R_DOWNR) b -= gn * (v[u] - (u + 1 < kRW ? v[u + 1 < kRW ? u + 1 : 0] : vno));
          if (f & R_DOWNL) b -= gl * (v[u] - vl);
          b += 2.0 * kdx;
          if (inj) b += 2.0 * iv.inp64[row];
        }
        rh[u] = b;
        const float bf = d2f(b);
        bacc += bf * bf;
        double rr = fma(-d, xv[u], b);
        if (f & R_UP) rr = fma(g[u], xmo, rr);
        if (f & R_DOWNR) rr = fma(gn, u + 1 < kRW ? xv[u + 1 < kRW ? u + 1 : 0] : xp, rr);
        if (f & R_DOWNL) rr = fma(gl, xl, rr);
        rr4[u] = d2f(rr);
        racc += rr * rr;
      }
      if (dense) {
        st_rows(gate + rb, g0);
        st_rows(gate + N + rb, g1);
        st_rows(gate + 2 * N + rb, g2);
      }
      st_rows(iv.diag + rb, dg);
      st_rows(iv.rhs + rb, rh);
      st_rows((float *)iv.cdiag + rb, cc);
      st_rows(c.w.Wb + rb, rr4);
    }
    r.ids(c, iv);
    window_maps(r, cc, gf, (Mob<float> *)iv.pmob + c.ip0, sc);
  }
  __syncthreads();  // its scans' scratch is free for the next reduction
  return make_double2((double)bacc, racc);
}

struct RefineX {
  float4 s, v;  // pstat, pval
  double2 b;    // the potential of the piece's first and last row before the update
};

// The walks of one refinement cycle, with the new potential of the pieces' first and last
// rows (in a group: of this CTA's pieces and the ones next to them).  pb: the buffer of the
// pieces' values.
template <int kMode>
__device__ __noinline__ void refine_walk(Ctx<float, kMode> c, int pb) {
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

// x += z by substitution (x0 = 2 Vin - Vout when Vin is not null, else Vout), then the FP64
// residual b - A x; returns the thread's part of ||scale r||^2 in FP32 (see ph_residual).
// kElim: eliminates r into buffer pb of the pieces' values; else stores it (W_0).
template <int kMode, bool kElim>
__device__ __noinline__ float refine_update(Ctx<float, kMode> c, const double *Vin, double *Vout,
                                            float scale, int pb) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<float> k = walk_of(c, iv, S);
  float *scz = (float *)S.warp, *sc0 = scz + 2 * kWarps, *sc1 = sc0 + 2 * kWarps;
  double *ends = S.warp + 4 * kWarps;
  float *pval = (float *)iv.pval + 4 * ((int64_t)c.ip0 + (int64_t)pb * iv.npieces);
  double *pxb = (double *)iv.pxb + 2 * ((int64_t)c.ip0 + (int64_t)pb * iv.npieces);
  float acc = 0;
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
      ld_rows((const double *)Vout + rb, x);
      if (Vin) {
        double v[kRW];
        ld_rows(Vin + rb, v);
#pragma unroll
        for (int u = 0; u < kRW; u++)
          if (!r.is(u, P_IDENT)) x[u] = 2.0 * v[u] - x[u];
      }
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
    affine_enter<float, 1, false>(A, M, scz, y);
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
  }
  __syncthreads();  // its scans' scratch is free for the next reduction
  return acc;
}

}  // namespace nrt
