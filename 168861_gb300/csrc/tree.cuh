// Exact tree preconditioner of the implicit kernel (included by implicit.cu after the
// kernel's context types).
//
// Factorisation of the whole tree matrix in Hines order (leaves to root), written for the
// input conductance eta of the subtree below each row: with d_k = g_k + eta_k (g_k the
// conductance to the mother, 0 on a row without that column),
//
//   eta_k = c_k + sum over children ch of g_ch eta_ch / (g_ch + eta_ch),
//
// which is d_k = D_k - sum g_ch^2 / d_ch rewritten without the cancellation between D_k and
// the children's terms (every term is positive), so the pivots keep full relative precision
// in FP32.  Per row: inv_k = 1 / d_k and e_k = g_k / d_k.  Solve: y_k = v_k + e y over the
// children, leaves to root, then z_k = inv_k y_k + e_k z_mother, root to leaves.
//
// Work is split into *pieces*: runs of consecutive rows in which each row's mother is the row
// before it, ended by branch points, sealed ends and window edges.  A window is ImView::win
// consecutive rows of an instance, kRW consecutive rows per thread of a CTA (at most 1024; fewer
// where a small tree's rows are to be spread over more SMs, and then the CTA's last warps have
// none); a piece lies in one window.  Everything a piece passes to the rest of the tree is a map of one number in,
// one number out, whatever the rest of the tree holds:
//   - factorisation: the conductance s that its children give its last row -> the
//     conductance e_f eta_f its first row gives its mother, a Moebius map (2x2 matrix);
//   - elimination: y entering its last row -> e_f y_f = A + B y;
//   - substitution: z_mother of its first row -> z of its last row = aL + bL y + B z_mother,
//     with B the product of the piece's e.
// So a sweep over the tree is three phases: every window finds its pieces' maps (segmented
// scans over the window, all windows in parallel), one CTA walks the pieces level by level
// (a few numbers per piece, in shared memory), and every window evaluates its rows.  Rows are
// read in row order with 16-byte loads, and all windows are full, whatever the branch
// structure; the number of levels only sets the length of the walk (about 0.1-0.3 us per
// level), not the number of passes over the rows or of grid-wide syncs (two per sweep; the
// level-by-level sweep that this replaces took one per level).
//
// In the solve the elimination runs with nothing entering each piece, giving alpha_k; with
// beta_k the product of e over the rows of the piece below k (once per factorisation),
// y_k = alpha_k + beta_k y_in, and the maps' remaining numbers are sums along the piece:
// aL = sum inv_k beta_k alpha_k, bL = sum inv_k beta_k^2.
#pragma once

namespace nrt {

// ---- the rows of one thread in a window

enum : uint8_t { P_IDENT = 1, P_UP = 2, P_FIRST = 32, P_LAST = 64 };  // ImView::pfl (with R_*)

// kRW values of this thread's rows; 16-byte loads and stores (row arrays are padded to
// multiples of kRW rows, instances start on one).
template <typename T>
__device__ __forceinline__ void ld_rows(const T *p, T (&o)[kRW]) {
  static_assert(kRW == 4, "vector widths below");
  if (sizeof(T) == 4) {
    const float4 v = *(const float4 *)(const void *)p;
    o[0] = (T)v.x; o[1] = (T)v.y; o[2] = (T)v.z; o[3] = (T)v.w;
  } else {
    const double2 a = ((const double2 *)(const void *)p)[0], b = ((const double2 *)(const void *)p)[1];
    o[0] = (T)a.x; o[1] = (T)a.y; o[2] = (T)b.x; o[3] = (T)b.y;
  }
}
template <typename T>
__device__ __forceinline__ void st_rows(T *p, const T (&o)[kRW]) {
  if (sizeof(T) == 4) {
    *(float4 *)(void *)p = make_float4((float)o[0], (float)o[1], (float)o[2], (float)o[3]);
  } else {
    ((double2 *)(void *)p)[0] = make_double2((double)o[0], (double)o[1]);
    ((double2 *)(void *)p)[1] = make_double2((double)o[2], (double)o[3]);
  }
}

// A window is the CTA's, or (iv.solo: windows of one warp's 128 rows) a warp's, which then takes
// every kWarps-th of its CTA's and has no barrier with the others in a pass.
__device__ __forceinline__ int window_thread(const ImView &iv) {
  return iv.solo ? (int)threadIdx.x & 31 : (int)threadIdx.x;
}
template <typename T, int kMode>
__device__ __forceinline__ int first_window(const Ctx<T, kMode> &c, const ImView &iv) {
  return c.w0 + (iv.solo ? (int)threadIdx.x >> 5 : 0);
}
__device__ __forceinline__ int window_stride(const ImView &iv) { return iv.solo ? kWarps : 1; }

// This thread's place in the arrays of one entry per thread of a window.
__device__ __forceinline__ int64_t thread_slot(const ImView &iv, int w) {
  return (int64_t)w * (iv.win / kRW) + window_thread(iv);
}

// This thread's rows of window w: first row, whether they belong to the instance, flags
// (rows that belong to no piece read as P_IDENT) and, after ids(), the id of each row's piece.
// ids() waits for the window's tables and makes a dependent load, so callers issue the loads
// of their rows before it.
template <typename T, int kMode>
struct WinRows {
  int64_t rb;
  bool ok, solo, idle;  // idle: no thread of this warp has rows in a window
  uint32_t q;
  int ord;   // ordinal (in row order) of the piece of the row before this thread's first
  int pid[kRW];
  __device__ __forceinline__ WinRows(const Ctx<T, kMode> &c, const ImView &iv, int w) {
    const int l = window_thread(iv) * kRW;
    rb = c.wrow0 + (int64_t)(w - c.iw0) * iv.win + l;
    ok = l < iv.win && rb < c.wend;
    solo = iv.solo;
    idle = !solo && ((int)threadIdx.x & ~31) * kRW >= iv.win;
    q = ok ? *(const uint32_t *)(iv.pfl + rb) : 0x01010101u * P_IDENT;
    ord = iv.wbase[w] - 1;
    if (ok) ord += (int)iv.wtp[thread_slot(iv, w)];
  }
  __device__ __forceinline__ bool is(int u, uint32_t flag) const { return (q >> (8 * u)) & flag; }
  __device__ __forceinline__ void ids(const Ctx<T, kMode> &c, const ImView &iv) {
    const int *map = iv.pmap + c.ip0;
#pragma unroll
    for (int u = 0; u < kRW; u++) {
      const bool first = is(u, P_FIRST);
      if (first) ord++;
      pid[u] = 0;
      if (!is(u, P_IDENT)) pid[u] = (u == 0 || first) ? map[ord] : pid[u > 0 ? u - 1 : 0];
    }
  }
};

// The initial guess x0 of a step, as refine_assemble leaves it for the passes that would form it
// again: a row's low word in Z_0, its high word in Z_1 (there are m + 1 >= 2 columns), at the
// row's own place.  Z is one workspace of all trees, a column ld rows apart, and trees run side by
// side: as an array of doubles x0 would lie on other trees' rows of Z_0 and Z_1, which one of them
// may be using for its GMRES basis.
template <typename T>
__device__ __forceinline__ void x0_store(T *Z, int64_t ld, int64_t row, double x) {
  static_assert(sizeof(T) == 4, "a word each");
  ((int *)(void *)Z)[row] = __double2loint(x);
  ((int *)(void *)Z)[ld + row] = __double2hiint(x);
}
template <typename T>
__device__ __forceinline__ double x0_load(const T *Z, int64_t ld, int64_t row) {
  if constexpr (sizeof(T) == 4) {
    const int *z = (const int *)(const void *)Z;
    return __hiloint2double(z[ld + row], z[row]);
  } else {
    return 0.0;  // FP64 steps keep no initial guess
  }
}
__device__ __forceinline__ void x0_rows(const float *Z, int64_t ld, int64_t rb, double (&x)[kRW]) {
  const int4 lo = *(const int4 *)(const void *)(Z + rb), hi = *(const int4 *)(const void *)(Z + ld + rb);
  x[0] = __hiloint2double(hi.x, lo.x);
  x[1] = __hiloint2double(hi.y, lo.y);
  x[2] = __hiloint2double(hi.z, lo.z);
  x[3] = __hiloint2double(hi.w, lo.w);
}

// ---- scans over the CTA's threads (every thread takes part)

// Value entering this thread's part of kN affine recurrences y <- A + M y that share M, in
// ascending or (kDesc) descending thread order, with 0 entering the first thread.
// sc: (kN + 1) * kWarps values.  One CTA barrier; a caller alternates between two scratch
// areas, so that the next scan's writes never meet this one's reads.  idle: the warp has no rows
// (its part is the identity and nobody reads its y).  solo: the scan is the warp's, without the
// barrier.
template <typename T, int kN, bool kDesc>
__device__ __forceinline__ void affine_enter(const T (&A)[kN], T M, T *sc, T (&y)[kN], bool idle,
                                             bool solo) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (idle) {
    if (lane == 0) {
      sc[w] = 1;
#pragma unroll
      for (int q = 0; q < kN; q++) sc[(q + 1) * kWarps + w] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kN; q++) y[q] = 0;
    return;
  }
  const int sl = kDesc ? 31 - lane : lane;  // position in scan order inside the warp
  T iA[kN], iM = M;
#pragma unroll
  for (int q = 0; q < kN; q++) iA[q] = A[q];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T pM = kDesc ? __shfl_down_sync(0xffffffffu, iM, off) : __shfl_up_sync(0xffffffffu, iM, off);
#pragma unroll
    for (int q = 0; q < kN; q++) {
      const T pA = kDesc ? __shfl_down_sync(0xffffffffu, iA[q], off)
                         : __shfl_up_sync(0xffffffffu, iA[q], off);
      if (sl >= off) iA[q] = iA[q] + iM * pA;
    }
    if (sl >= off) iM = iM * pM;
  }
  T eA[kN];
  T eM = kDesc ? __shfl_down_sync(0xffffffffu, iM, 1) : __shfl_up_sync(0xffffffffu, iM, 1);
#pragma unroll
  for (int q = 0; q < kN; q++)
    eA[q] = kDesc ? __shfl_down_sync(0xffffffffu, iA[q], 1) : __shfl_up_sync(0xffffffffu, iA[q], 1);
  if (solo) {
#pragma unroll
    for (int q = 0; q < kN; q++) y[q] = sl == 0 ? (T)0 : eA[q];
    return;
  }
  if (sl == 31) {
    sc[w] = iM;
#pragma unroll
    for (int q = 0; q < kN; q++) sc[(q + 1) * kWarps + w] = iA[q];
  }
  if (sl == 0) {
    eM = 1;
#pragma unroll
    for (int q = 0; q < kN; q++) eA[q] = 0;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kN; q++) {
    T v = 0;
    if (kDesc) {
      for (int p = kWarps - 1; p > w; p--) v = sc[(q + 1) * kWarps + p] + sc[p] * v;
    } else {
      for (int p = 0; p < w; p++) v = sc[(q + 1) * kWarps + p] + sc[p] * v;
    }
    y[q] = eA[q] + eM * v;
  }
}

// 2x2 matrices of the pivot recurrence (non-negative entries), scaled by powers of two.
template <typename T>
struct Mob {
  T a, b, c, d;  // [[a, b], [c, d]]
};

__device__ __forceinline__ float quot(float a, float b) { return a / b; }
__device__ __forceinline__ double quot(double a, double b) { return div64(a, b); }

// 2^e, e in the exponent's normal range.
template <typename T>
__device__ __forceinline__ T pow2_of(int e) {
  if constexpr (sizeof(T) == 4) return __int_as_float((e + 127) << 23);
  else return __hiloint2double((e + 1023) << 20, 0);
}

// A power of two near 1 / m for a positive normal m.
__device__ __forceinline__ float pow2_near_inv(float m) {
  const int e = (__float_as_int(m) >> 23) & 255;
  return __int_as_float(max(254 - e, 1) << 23);
}
__device__ __forceinline__ double pow2_near_inv(double m) {
  const int e = (__double2hiint(m) >> 20) & 2047;
  return __hiloint2double(max(2046 - e, 1) << 20, 0);
}

template <typename T>
__device__ __forceinline__ T max_of(T a, T b) {
  return a > b ? a : b;
}

// Scales the numbers by one power of two so that the largest lies in [1, 2) (FP32: [1, 4)).  In
// FP64 on the exponents, in integers: a comparison or a product of doubles takes an SM's FP64 pipe
// 16 cycles, and of a matrix product's 15 such operations 7 were its scaling (48 trees of 1e3 to 1e4 in
// FP64, 8 steps: 2.31 -> 2.17 ms).  What would leave
// the range is 0, as far below the largest as 2^-1022; a largest number that is no positive normal
// one (0, infinite, NaN, or a negative entry among them) takes the general way.
template <int kN>
__device__ __forceinline__ void scale_to_one(float (&x)[kN]) {
  float m = x[0];
#pragma unroll
  for (int i = 1; i < kN; i++) m = max_of(m, x[i]);
  const float s = pow2_near_inv(m);
#pragma unroll
  for (int i = 0; i < kN; i++) x[i] *= s;
}
template <int kN>
__device__ __forceinline__ void scale_to_one(double (&x)[kN]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < kN; i++) m = max(m, (uint32_t)__double2hiint(x[i]));
  const uint32_t e = m >> 20;
  if (e - 1u >= 2046u) {
    double big = x[0];
#pragma unroll
    for (int i = 1; i < kN; i++) big = max_of(big, x[i]);
    const double s = pow2_near_inv(big);
#pragma unroll
    for (int i = 0; i < kN; i++) x[i] *= s;
    return;
  }
  const uint32_t low = (e > 1023u ? e - 1022u : 1u) << 20, d = (1023u - e) << 20;
#pragma unroll
  for (int i = 0; i < kN; i++) {
    const uint32_t h = (uint32_t)__double2hiint(x[i]);
    x[i] = h >= low ? __hiloint2double((int)(h + d), __double2loint(x[i])) : 0.0;
  }
}

template <typename T>
__device__ __forceinline__ Mob<T> mob_scaled(const Mob<T> &r) {
  T x[4] = {r.a, r.b, r.c, r.d};
  scale_to_one(x);
  return Mob<T>{x[0], x[1], x[2], x[3]};
}

template <typename T>
__device__ __forceinline__ Mob<T> mob_mul(const Mob<T> &x, const Mob<T> &y) {  // x * y
  return mob_scaled(Mob<T>{x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d,
                           x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d});
}

// The map of one row after P: a vector (a, b), a / b the conductance that the rows below give
// this one, becomes (g p, p + g b) with p = a + c b.
template <typename T>
__device__ __forceinline__ Mob<T> mob_row(T c, T g, const Mob<T> &P) {
  const T pa = P.a + c * P.c, pb = P.b + c * P.d;
  return mob_scaled(Mob<T>{g * pa, g * pb, pa + g * P.c, pb + g * P.d});
}

template <typename T>
__device__ __forceinline__ Mob<T> mob_shfl_down(const Mob<T> &m, int off) {
  return Mob<T>{__shfl_down_sync(0xffffffffu, m.a, off), __shfl_down_sync(0xffffffffu, m.b, off),
                __shfl_down_sync(0xffffffffu, m.c, off), __shfl_down_sync(0xffffffffu, m.d, off)};
}

// ---- the walk over the pieces (one CTA)

// The numbers of the walk, one per piece of the instance (ids in level order, deepest first).
// A CTA alone with many pieces keeps the first four in shared memory (or in device memory
// when there are too many) and loads each level's maps and links one level ahead.  In a group
// every CTA walks all pieces redundantly, with the maps and links staged in shared memory as well: the
// levels of a bushy tree hold a thousand pieces, and a walk that loads them level by level took
// 10 to 17 us (2,937 pieces on 14 levels) where the staged one takes 3 to 4.
template <typename T>
struct Walk {
  double2 *px;    // refinement updates: the potential of its first and last row after the update
  T *val;         // what the piece passes on: up (to its mother's piece), then z of its last row
  T *yin;         // what enters its last row (factorisation: the children's conductance)
  T *zpar;        // z of its first row's mother
  Mob<T> *st;     // staged: its matrix, or B, bL, A, aL
  ushort4 *link;  // staged: plink (65535: none)
};

constexpr int kNoPiece = 65535;

// Bytes of the walk's numbers per piece.
__host__ __device__ constexpr size_t walk_bytes(size_t tb, bool staged) {
  return 16 + 3 * tb + (staged ? 4 * tb + 8 : 0);
}

template <typename T, int kMode>
__device__ __forceinline__ Walk<T> walk_of(const Ctx<T, kMode> &c, const ImView &iv, const Shared &S) {
  Walk<T> k;
  if (c.np <= iv.walk_cap) {
    const int ns = c.np <= iv.stage_cap ? c.np : 0;
    k.px = (double2 *)S.tile;
    k.st = (Mob<T> *)(k.px + c.np);
    k.link = (ushort4 *)(k.st + ns);
    k.val = (T *)(k.link + ns);
  } else {  // all instances' potentials, then all instances' numbers: each array aligned
    k.px = (double2 *)iv.gwalk + c.ip0;
    k.st = nullptr;
    k.link = nullptr;
    k.val = (T *)((double2 *)iv.gwalk + iv.npieces) + 3 * (int64_t)c.ip0;
  }
  k.yin = k.val + c.np;
  k.zpar = k.yin + c.np;
  return k;
}

// Whether this CTA walks: its own instance (block), or every CTA of the group redundantly
// when the walk's numbers fit its shared memory, else the group's first.
template <typename T, int kMode>
__device__ __forceinline__ bool walks(const Ctx<T, kMode> &c, const ImView &iv) {
  return one_cta(kMode) || c.np <= iv.walk_cap || c.rank == 0;
}
// Whether the maps and links of this walk are staged: in a group all that fit, in a block those
// of few pieces (one warp's windows cut a long cable into a chain of them, and a level that waits
// for device memory takes 1 us).
template <typename T, int kMode>
__device__ __forceinline__ bool staged(const Ctx<T, kMode> &c, const ImView &iv) {
  return c.np <= iv.stage_cap;
}

// The links of the instance, staged once per launch.
template <typename T, int kMode>
__device__ __noinline__ void stage_links(const Ctx<T, kMode> &c) {
  const ImView &iv = *c.iv;
  if (!staged(c, iv)) return;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<T> k = walk_of(c, iv, S);
#pragma unroll 4
  for (int q = threadIdx.x; q < c.np; q += kThreads) {
    const int4 l = iv.plink[c.ip0 + q];
    k.link[q] = make_ushort4((unsigned short)l.x, (unsigned short)l.y, (unsigned short)l.z,
                             (unsigned short)l.w);
  }
  __syncthreads();
}

// Up-walk: f(x, children's sum) -> what the piece passes on, x = get(piece id).
template <typename T, int kMode, typename X, typename Get, typename F>
__device__ __forceinline__ void walk_up(const Ctx<T, kMode> &c, const ImView &iv, Walk<T> k,
                                        Get get, F f) {
  const int *lo = c.lev;
  const int nl = c.l1 - c.l0;
  if (staged(c, iv)) {
    int qb = 0, qe = lo[0];
    for (int e = 0; e < nl; e++) {
      const int qn = e + 1 < nl ? lo[e + 1] : 0;
      for (int q = qb + threadIdx.x; q < qe; q += kThreads) {
        const ushort4 t = k.link[q];
        const T s = (t.x != kNoPiece ? k.val[t.x] : (T)0) + (t.y != kNoPiece ? k.val[t.y] : (T)0);
        k.yin[q] = s;
        k.val[q] = f(get(q), s);
      }
      __syncthreads();
      qb = qe;
      qe = qn;
    }
    return;
  }
  const int4 *lk = iv.plink + c.ip0;
  int qb = 0, qe = lo[0], q = threadIdx.x;
  int4 t = make_int4(-1, -1, -1, 0);
  X x{};
  if (q < qe) {
    t = lk[q];
    x = get(q);
  }
  for (int e = 0; e < nl; e++) {
    const int qe2 = e + 1 < nl ? lo[e + 1] : qe, qn = qe + (int)threadIdx.x;
    int4 tn = make_int4(-1, -1, -1, 0);
    X xn{};
    if (qn < qe2) {
      tn = lk[qn];
      xn = get(qn);
    }
    for (q = qb + threadIdx.x; q < qe; q += kThreads) {
      if (q >= qb + kThreads) {
        t = lk[q];
        x = get(q);
      }
      const T s = (t.x >= 0 ? k.val[t.x] : (T)0) + (t.y >= 0 ? k.val[t.y] : (T)0);
      k.yin[q] = s;
      k.val[q] = f(x, s);
    }
    __syncthreads();
    t = tn;
    x = xn;
    qb = qe;
    qe = qe2;
  }
}

// Down-walk: f(piece id, x, yin, z of the mother) -> z of the piece's last row.
template <typename T, int kMode, typename X, typename Get, typename F>
__device__ __forceinline__ void walk_down(const Ctx<T, kMode> &c, const ImView &iv, Walk<T> k,
                                          Get get, F f) {
  const int *lo = c.lev;
  const int nl = c.l1 - c.l0;
  int qe = nl > 0 ? lo[nl - 1] : 0, qb = nl > 1 ? lo[nl - 2] : 0;
  if (staged(c, iv)) {
    for (int e = nl - 1; e >= 0; e--) {
      const int qp = e > 1 ? lo[e - 2] : 0;
      for (int q = qb + threadIdx.x; q < qe; q += kThreads) {
        const int par = k.link[q].z;
        const T zp = par != kNoPiece ? k.val[par] : (T)0;
        k.zpar[q] = zp;
        k.val[q] = f(q, get(q), k.yin[q], zp);
      }
      __syncthreads();
      qe = qb;
      qb = qp;
    }
    return;
  }
  const int4 *lk = iv.plink + c.ip0;
  int par = -1;
  X x{};
  if (qb + (int)threadIdx.x < qe) {
    par = lk[qb + threadIdx.x].z;
    x = get(qb + threadIdx.x);
  }
  for (int e = nl - 1; e >= 0; e--) {
    const int qp = e > 1 ? lo[e - 2] : 0;
    int parn = -1;
    X xn{};
    if (e > 0 && qp + (int)threadIdx.x < qb) {
      parn = lk[qp + threadIdx.x].z;
      xn = get(qp + threadIdx.x);
    }
    for (int q = qb + threadIdx.x; q < qe; q += kThreads) {
      if (q >= qb + kThreads) {
        par = lk[q].z;
        x = get(q);
      }
      const T zp = par >= 0 ? k.val[par] : (T)0;
      k.zpar[q] = zp;
      k.val[q] = f(q, x, k.yin[q], zp);
    }
    __syncthreads();
    par = parn;
    x = xn;
    qe = qb;
    qb = qp;
  }
}

// ---- factorisation

// The 2x2 matrices of the pieces of one window: cc, g the thread's rows (g changed to 0 on
// rows without a mother column).  ent: the thread's place for the map of the rows of its last
// row's piece that later threads hold, which tree_pivots starts from.  sc: 5 * kWarps values; one
// CTA barrier.
template <typename T, int kMode>
__device__ __forceinline__ void window_maps(const WinRows<T, kMode> &r, const T (&cc)[kRW],
                                            T (&g)[kRW], Mob<T> *out, T *ent, T *sc) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const Mob<T> one{1, 0, 0, 1};
  if (r.idle) {
    if (lane == 0) {
      sc[wp] = sc[3 * kWarps + wp] = 1;
      sc[kWarps + wp] = sc[2 * kWarps + wp] = sc[4 * kWarps + wp] = 0;
    }
    __syncthreads();
    return;
  }
  // rows in descending order; a piece's last row starts its matrix afresh
  Mob<T> P = one;
  bool R = false;
#pragma unroll
  for (int u = kRW - 1; u >= 0; u--) {
    if (r.is(u, P_IDENT)) continue;
    if (!(r.is(u, P_UP))) g[u] = 0;
    if (r.is(u, P_LAST)) {
      P = one;
      R = true;
    }
    P = mob_row(cc[u], g[u], P);
  }
  Mob<T> I = P;
  bool IR = R;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const Mob<T> Q = mob_shfl_down(I, off);
    const bool qR = __shfl_down_sync(0xffffffffu, (int)IR, off) != 0;
    if (31 - lane >= off && !IR) {
      I = mob_mul(I, Q);
      IR = qR;
    }
  }
  Mob<T> E = mob_shfl_down(I, 1);
  bool ER = __shfl_down_sync(0xffffffffu, (int)IR, 1) != 0;
  if (lane == 31) {
    E = one;
    ER = false;
  }
  if (!r.solo) {
    if (lane == 0) {
      sc[wp] = I.a;
      sc[kWarps + wp] = I.b;
      sc[2 * kWarps + wp] = I.c;
      sc[3 * kWarps + wp] = I.d;
      sc[4 * kWarps + wp] = IR ? (T)1 : (T)0;
    }
    __syncthreads();
  }
  if (!r.solo && !ER && !(r.is(kRW - 1, P_LAST))) {  // this thread continues an earlier warp's piece
    Mob<T> X = one;
    int p = wp + 1;
    while (p < kWarps && sc[4 * kWarps + p] == (T)0) p++;
    for (p = min(p, kWarps - 1); p > wp; p--)
      X = mob_mul(Mob<T>{sc[p], sc[kWarps + p], sc[2 * kWarps + p], sc[3 * kWarps + p]}, X);
    E = mob_mul(E, X);
  }
  if (r.ok) {
    const T e4[4] = {E.a, E.b, E.c, E.d};
    st_rows(ent, e4);
  }
  Mob<T> cur = E;
#pragma unroll
  for (int u = kRW - 1; u >= 0; u--) {
    if (r.is(u, P_IDENT)) continue;
    if (r.is(u, P_LAST)) cur = one;
    cur = mob_row(cc[u], g[u], cur);
    if (r.is(u, P_FIRST)) out[r.pid[u]] = cur;
  }
}

template <typename T, int kMode>
__device__ __noinline__ void tree_maps(const Ctx<T, kMode> &c) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const T *C = (const T *)iv.cdiag;
  const T *G = sizeof(T) == 4 ? (const T *)(const void *)iv.gf : (const T *)(const void *)iv.g64;
  int par = 0;
  for (int w = first_window(c, iv); w < c.w1; w += window_stride(iv)) {
    T *sc = (T *)S.warp + par * 5 * kWarps;
    par ^= 1;
    WinRows<T, kMode> r(c, iv, w);
    T cc[kRW] = {}, g[kRW] = {};
    if (r.ok) {
      ld_rows(C + r.rb, cc);
      ld_rows(G + r.rb, g);
    }
    r.ids(c, iv);
    window_maps(r, cc, g, (Mob<T> *)iv.pmob + c.ip0,
                (T *)iv.tent + 4 * thread_slot(iv, w), sc);
  }
}

// Pivots from the children's conductances: inv, e, beta of every row, and per piece the
// product B of its e and bL.  The rows of v, the first right-hand side, are eliminated in the
// same pass (tree_eliminate, into buffer 0 of the pieces' values).  ends: the initial guess of each
// piece's first and last row is exported too, for the refinement's updates.
template <typename T, int kMode>
__device__ __noinline__ void tree_pivots(const Ctx<T, kMode> &c, const T *v, bool ends) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<T> k = walk_of(c, iv, S);
  const T *C = (const T *)iv.cdiag;
  const T *G = sizeof(T) == 4 ? (const T *)(const void *)iv.gf : (const T *)(const void *)iv.g64;
  T *pstat = (T *)iv.pstat + 4 * (int64_t)c.ip0, *pval = (T *)iv.pval + 4 * (int64_t)c.ip0;
  double *pxb = (double *)iv.pxb + 2 * (int64_t)c.ip0;
  for (int w = first_window(c, iv); w < c.w1; w += window_stride(iv)) {
    T *sc1 = (T *)S.warp, *sc2 = sc1 + 3 * kWarps;
    WinRows<T, kMode> r(c, iv, w);
    T cc[kRW] = {}, g[kRW] = {}, al[kRW] = {}, en[4] = {1, 0, 0, 1};
    if (r.ok) {
      ld_rows((const T *)iv.tent + 4 * thread_slot(iv, w), en);
      ld_rows(C + r.rb, cc);
      ld_rows(G + r.rb, g);
      ld_rows(v + r.rb, al);
    }
    r.ids(c, iv);
    // the vector entering the thread's last row: its piece's (s, 1) through the later rows
    T va = 0, vb = 1;
    if (!r.idle) {
      const T s = k.yin[r.pid[kRW - 1]];
      const T na = en[0] * s + en[1], nb = en[2] * s + en[3];
      T n2[2] = {na, nb};
      scale_to_one(n2);
      va = n2[0];
      vb = n2[1];
    }
    T inv[kRW], ee[kRW], beta[kRW];
    // what a row passes on: beta u <- e u with 1 entering each piece's last row, alpha
    // u <- e (v + u) with 0
    T A[2] = {0, 0}, M = 1;
#pragma unroll
    for (int u = kRW - 1; u >= 0; u--) {
      inv[u] = 0;
      ee[u] = 0;
      if (r.is(u, P_IDENT)) continue;
      if (!(r.is(u, P_UP))) g[u] = 0;
      if (r.is(u, P_LAST)) {
        va = k.yin[r.pid[u]];
        vb = 1;
      }
      // eta = p / vb; the pivot g + eta = (p + g vb) / vb
      const T p = va + cc[u] * vb;
      const T na = g[u] * p, nb = p + g[u] * vb;
      inv[u] = quot(vb, nb);
      ee[u] = g[u] * inv[u];
      T n2[2] = {na, nb};
      scale_to_one(n2);
      va = n2[0];
      vb = n2[1];
      if (r.is(u, P_LAST)) {
        A[0] = ee[u];
        A[1] = ee[u] * al[u];
        M = 0;
      } else {
        A[0] *= ee[u];
        A[1] = ee[u] * (al[u] + A[1]);
        M *= ee[u];
      }
    }
    T y[2];
    affine_enter<T, 2, true>(A, M, sc1, y, r.idle, r.solo);
    T sb[2] = {0, 0}, sm = 1, cur = y[0], cua = y[1];
#pragma unroll
    for (int u = kRW - 1; u >= 0; u--) {
      beta[u] = 0;
      if (r.is(u, P_IDENT)) {
        al[u] = 0;
        continue;
      }
      beta[u] = (r.is(u, P_LAST)) ? (T)1 : cur;
      if (!r.is(u, P_LAST)) al[u] += cua;
      cur = ee[u] * beta[u];
      cua = ee[u] * al[u];
      if (r.is(u, P_FIRST)) {
        T *ps = pstat + 4 * (int64_t)r.pid[u], *pa = pval + 4 * (int64_t)r.pid[u];
        ps[0] = cur;  // B
        ps[2] = inv[u] * beta[u];
        ps[3] = ee[u];
        pa[0] = cua;  // A
        pa[2] = inv[u] * al[u];
        if (ends) pxb[2 * (int64_t)r.pid[u]] = x0_load(c.w.Z, iv.ld, r.rb + u);
      }
    }
#pragma unroll
    for (int u = 0; u < kRW; u++) {
      if (r.is(u, P_FIRST)) sb[0] = sb[1] = sm = 0;
      const T wb = inv[u] * beta[u];
      sb[0] += wb * beta[u];
      sb[1] += wb * al[u];
    }
    affine_enter<T, 2, false>(sb, sm, sc2, y, r.idle, r.solo);
#pragma unroll
    for (int u = 0; u < kRW; u++) {
      if (r.is(u, P_FIRST)) y[0] = y[1] = 0;
      const T wb = inv[u] * beta[u];
      y[0] += wb * beta[u];
      y[1] += wb * al[u];
      if (r.is(u, P_LAST)) {
        pstat[4 * (int64_t)r.pid[u] + 1] = y[0];  // bL
        pval[4 * (int64_t)r.pid[u] + 1] = y[1];   // aL
        if (ends) pxb[2 * (int64_t)r.pid[u] + 1] = x0_load(c.w.Z, iv.ld, r.rb + u);
      }
    }
    if (r.ok) {
      st_rows((T *)iv.tinv + r.rb, inv);
      st_rows((T *)iv.te + r.rb, ee);
      st_rows((T *)iv.tbeta + r.rb, beta);
      st_rows((T *)iv.talpha + r.rb, al);
    }
  }
}

template <typename T, int kMode>
__device__ __noinline__ void walk_factor(const Ctx<T, kMode> &c) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<T> k = walk_of(c, iv, S);
  const Mob<T> *mob = (const Mob<T> *)iv.pmob + c.ip0;
  auto f = [](const Mob<T> &m, T s) { return quot(m.a * s + m.b, m.c * s + m.d); };
  if (staged(c, iv)) {
#pragma unroll 4
    for (int q = threadIdx.x; q < c.np; q += kThreads) k.st[q] = mob[q];
    __syncthreads();
    walk_up<T, kMode, Mob<T>>(c, iv, k, [&](int q) { return k.st[q]; }, f);
  } else {
    walk_up<T, kMode, Mob<T>>(c, iv, k, [&](int q) { return mob[q]; }, f);
  }
}

// The factorisation once every piece's matrix is known (tree_maps, or the windowed assembly)
// and visible to the walk.
template <typename T, int kMode>
__device__ __noinline__ void tree_factor(const Ctx<T, kMode> &c, const T *v, bool ends) {
  const ImView &iv = *c.iv;
  if (walks(c, iv)) walk_factor(c);
  if (!one_cta(kMode) && c.np > iv.walk_cap) group_sync<kMode>();
  tree_pivots(c, v, ends);
  __syncthreads();  // its scans' scratch is free for the next reduction
}

// ---- solve

// Elimination of one window with nothing entering the pieces: al = v in, alpha out; exports
// each piece's A = e_f alpha_f, aL and inv_f alpha_f.  sc0, sc1: 2 * kWarps values each; two
// CTA barriers.
template <typename T, int kMode>
__device__ __forceinline__ void window_eliminate(const WinRows<T, kMode> &r, T (&al)[kRW],
                                                 const T (&ee)[kRW], const T (&inv)[kRW],
                                                 const T (&be)[kRW], T *pval, T *sc0, T *sc1) {
  T A[1] = {0}, M = 1, y[1];
#pragma unroll
  for (int u = kRW - 1; u >= 0; u--) {
    if (r.is(u, P_IDENT)) {
      al[u] = 0;
      continue;
    }
    if (r.is(u, P_LAST)) {
      A[0] = ee[u] * al[u];
      M = 0;
    } else {
      A[0] = ee[u] * (al[u] + A[0]);
      M *= ee[u];
    }
  }
  affine_enter<T, 1, true>(A, M, sc0, y, r.idle, r.solo);
  T cur = y[0];
#pragma unroll
  for (int u = kRW - 1; u >= 0; u--) {
    if (r.is(u, P_IDENT)) continue;
    if (!r.is(u, P_LAST)) al[u] += cur;
    cur = ee[u] * al[u];
    if (r.is(u, P_FIRST)) {
      pval[4 * (int64_t)r.pid[u]] = cur;  // A
      pval[4 * (int64_t)r.pid[u] + 2] = inv[u] * al[u];
    }
  }
  T sb[1] = {0}, sm = 1;
#pragma unroll
  for (int u = 0; u < kRW; u++) {
    if (r.is(u, P_FIRST)) sb[0] = sm = 0;
    sb[0] += inv[u] * be[u] * al[u];
  }
  affine_enter<T, 1, false>(sb, sm, sc1, y, r.idle, r.solo);
#pragma unroll
  for (int u = 0; u < kRW; u++) {
    if (r.is(u, P_FIRST)) y[0] = 0;
    y[0] += inv[u] * be[u] * al[u];
    if (r.is(u, P_LAST)) pval[4 * (int64_t)r.pid[u] + 1] = y[0];  // aL
  }
}

// alpha of every row and the pieces' values for the right-hand side v.  pb: the buffer of the
// pieces' values; x (with Vin null) the potential whose first and last rows are exported.
template <typename T, int kMode>
__device__ __noinline__ void tree_eliminate(const Ctx<T, kMode> &c, const T *v, int pb, const double *x) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  T *pval = (T *)iv.pval + 4 * ((int64_t)c.ip0 + (int64_t)pb * iv.npieces);
  double *pxb = (double *)iv.pxb + 2 * ((int64_t)c.ip0 + (int64_t)pb * iv.npieces);
  T *sc0 = (T *)S.warp, *sc1 = sc0 + 2 * kWarps;
  for (int w = first_window(c, iv); w < c.w1; w += window_stride(iv)) {
    WinRows<T, kMode> r(c, iv, w);
    T al[kRW] = {}, ee[kRW] = {}, inv[kRW] = {}, be[kRW] = {};
    if (r.ok) {
      ld_rows(v + r.rb, al);
      ld_rows((const T *)iv.te + r.rb, ee);
      ld_rows((const T *)iv.tinv + r.rb, inv);
      ld_rows((const T *)iv.tbeta + r.rb, be);
    }
    r.ids(c, iv);
    if (x) {
#pragma unroll
      for (int u = 0; u < kRW; u++) {
        if (r.is(u, P_FIRST)) pxb[2 * (int64_t)r.pid[u]] = x[r.rb + u];
        if (r.is(u, P_LAST)) pxb[2 * (int64_t)r.pid[u] + 1] = x[r.rb + u];
      }
    }
    window_eliminate(r, al, ee, inv, be, pval, sc0, sc1);
    if (r.ok) st_rows((T *)iv.talpha + r.rb, al);
  }
}

// The solve's walks: a piece's numbers travel as Mob {B, bL, A, aL}.

template <typename T, int kMode>
__device__ __noinline__ void walk_solve(const Ctx<T, kMode> &c) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<T> k = walk_of(c, iv, S);
  const T *ps = (const T *)iv.pstat + 4 * (int64_t)c.ip0, *pa = (const T *)iv.pval + 4 * (int64_t)c.ip0;
  auto up = [](const Mob<T> &x, T s) { return x.c + x.a * s; };
  auto down = [](int, const Mob<T> &x, T y, T zp) { return x.d + x.b * y + x.a * zp; };
  auto get = [&](int q) { return Mob<T>{ps[4 * q], ps[4 * q + 1], pa[4 * q], pa[4 * q + 1]}; };
  if (staged(c, iv)) {
#pragma unroll 4
    for (int q = threadIdx.x; q < c.np; q += kThreads) k.st[q] = get(q);
    __syncthreads();
    auto sget = [&](int q) { return k.st[q]; };
    walk_up<T, kMode, Mob<T>>(c, iv, k, sget, up);
    walk_down<T, kMode, Mob<T>>(c, iv, k, sget, down);
  } else {
    walk_up<T, kMode, Mob<T>>(c, iv, k, get, up);
    walk_down<T, kMode, Mob<T>>(c, iv, k, get, down);
  }
}

// Substitution: z of every row (identity rows 0).
template <typename T, int kMode>
__device__ __noinline__ void tree_substitute(const Ctx<T, kMode> &c, T *z) {
  const ImView &iv = *c.iv;
  Shared S = carve(dyn_smem(), iv.m);
  const Walk<T> k = walk_of(c, iv, S);
  int par = 0;
  for (int w = first_window(c, iv); w < c.w1; w += window_stride(iv)) {
    T *sc = (T *)S.warp + par * 2 * kWarps;
    par ^= 1;
    WinRows<T, kMode> r(c, iv, w);
    T al[kRW] = {}, ee[kRW] = {}, inv[kRW] = {}, be[kRW] = {};
    if (r.ok) {
      ld_rows((const T *)iv.talpha + r.rb, al);
      ld_rows((const T *)iv.te + r.rb, ee);
      ld_rows((const T *)iv.tinv + r.rb, inv);
      ld_rows((const T *)iv.tbeta + r.rb, be);
    }
    r.ids(c, iv);
    T A[1] = {0}, M = 1, y[1];
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
    affine_enter<T, 1, false>(A, M, sc, y, r.idle, r.solo);
    T cur = y[0];
#pragma unroll
    for (int u = 0; u < kRW; u++) {
      if (r.is(u, P_IDENT)) {
        al[u] = 0;
        continue;
      }
      if (!(r.is(u, P_FIRST))) al[u] += ee[u] * cur;
      cur = al[u];
    }
    if (r.ok) st_rows(z + r.rb, al);
  }
}

// z = A^-1 v (up to rounding) with the factors of tree_factor.  eliminated: v is the
// right-hand side that tree_factor has eliminated.
template <typename T, int kMode>
__device__ __noinline__ void tree_apply(const Ctx<T, kMode> &c, const T *v, T *z, bool eliminated) {
  const ImView &iv = *c.iv;
  if (!eliminated) tree_eliminate(c, v, 0, (const double *)nullptr);
  group_sync<kMode>();
  if (walks(c, iv)) walk_solve(c);
  if (!one_cta(kMode) && c.np > iv.walk_cap) group_sync<kMode>();
  tree_substitute(c, z);
  __syncthreads();  // the walk's numbers are read before the next walk writes them
}

}  // namespace nrt
