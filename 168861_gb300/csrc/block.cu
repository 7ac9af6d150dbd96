// Several explicit steps per launch: tiles with halos.
//
// A step of the per-step kernels moves every element's state through memory (about 64 B) and
// ends with a launch boundary, and what it computes per element is small: a pack in L2 is bound
// by launches (a myelinated axon's 199,202 compartments took 6.4 us per step with its strain,
// 100,000 compartments in 24 trees 5.0 us), and a large batch by memory and by the instructions
// that load, unpack and store (22 million compartments 320 us per step, 75% of the copy
// bandwidth on its compulsory bytes).  Here a CTA loads a tile's state once, into registers,
// and advances it `depth` steps; only the FP32 potential passes between threads, through shared
// memory, one CTA barrier per step.  A tile's results depend on elements up to `depth` away:
// its halo, whose elements it advances as well, each while its value still reaches an owned
// element (distance <= steps left).  The arithmetic per element is explicit_step_mixed's,
// operation for operation, so every result is the per-step kernels' bit for bit.  FP64 packs
// have a form of their own (explicit_block_f64).
//
// Ownership: state is read from one set of buffers and written to another (potential, shadow
// and gates), because neighbouring tiles read an element's old state as their halo.
//
// Tiles are ranges of the element order (depth-first), so a halo is the few elements before
// and after the range along the cable plus, per branch whose two sides fall into different
// tiles, as many along it.  The plan is the host's (build_block_plan).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "block.h"
#include "cvt.cuh"
#include "hh.cuh"
#include "pdl.cuh"
#include "record.cuh"
#include "strain.cuh"

namespace nrt {

namespace {

// Recording after a launch's steps: one thread replays record_probe's rule over a probe's
// values (v[k * stride] after loop index i0 + k, n of them).
__device__ __forceinline__ void record_trace(const RecView &r, int slot, int64_t i0, int n,
                                             const double *v, int stride, double dT) {
  if (n <= 0) return;
  int32_t nspike = r.nspike[slot];
  int64_t prev_i = r.prev_i[slot], nsamp = r.nsamp[slot];
  double prev_v = r.prev_v[slot];
  // the first loop index >= i0 that is sampled: i - origin + 1 a positive multiple of m
  const int64_t m = r.interval + 1, q = i0 - r.origin + 1;
  int64_t s = q <= 0 ? 0 : (q + m - 1) / m - 1;  // its sample number
  int64_t next = r.origin - 1 + (s + 1) * m;
  for (int k = 0; k < n; k++) {
    const int64_t i = i0 + k;
    const double x = v[k * stride];
    if (prev_i == i - 1 && prev_v < r.thresh && x >= r.thresh) {
      if (nspike < r.max_spikes) {
        const double t0 = (double)(i - 1) * dT, t1 = (double)i * dT;
        const double frac = (r.thresh - prev_v) * (t1 - t0);
        r.spk[(int64_t)slot * r.max_spikes + nspike] = t0 + frac / (x - prev_v);
      }
      nspike++;
    }
    prev_v = x;
    prev_i = i;
    if (i == next) {
      if (s < r.cap) r.val[(int64_t)slot * r.cap + s] = x;
      if (s + 1 > nsamp) nsamp = s + 1;
      s++;
      next += m;
    }
  }
  r.nspike[slot] = nspike;
  r.prev_i[slot] = prev_i;
  r.prev_v[slot] = prev_v;
  r.nsamp[slot] = nsamp;
}

__device__ __forceinline__ int clip_int(int64_t x) {
  return x > 1 << 30 ? 1 << 30 : (x < -(1 << 30) ? -(1 << 30) : (int)x);
}

// Every probe of a tile from the trace (complete: the last step ended with a barrier).
__device__ __forceinline__ void record_tile(const PackView &p, const BlockView &bv,
                                            const BlockTile &t, const RecView &r, int k0, int nk,
                                            const double *trace, int np) {
  for (int e = threadIdx.x; e < np; e += blockDim.x) {
    const int2 x = bv.probe[t.p0 + e];
    int c0 = e;  // the column of the element's first probe
    for (int u = 0; u < e; u++)
      if (bv.probe[t.p0 + u].x == x.x) {
        c0 = u;
        break;
      }
    const InstDev in = p.inst[r.inst[x.y]];
    record_trace(r, x.y, in.base + k0, min(nk, clip_int(in.iend - in.base - k0)), trace + c0, np,
                 in.dT);
  }
}

// One thread per local element.  kDense (most elements are HH): the channel parameters stay in
// registers, 64 per thread; otherwise HH elements read them every step and 40 registers leave
// room for 1536 threads on an SM, which a myelinated axon of 200,000 compartments needs to be
// resident at once.
template <bool kDense, bool kStrain, bool kRec>
__global__ void __launch_bounds__(kDense ? 512 : 256, kDense ? 2 : 6)
    explicit_block_mixed(PackView p, BlockView bv, int k0, int nk, const double *Vin, double *Vout,
                         float *Fout, const float *gin, float *gout, RecView r, StrainView sv) {
  extern __shared__ __align__(16) unsigned char bsm[];
  float *F = (float *)bsm;                       // [2][cap]
  float *G = F + 2 * bv.cap;                     // [kStrain ? 2 : 1][cap]
  ushort4 *nb = (ushort4 *)(G + (kStrain ? 2 : 1) * bv.cap);  // [cap] {mother, DR, DL, -}
  float *rows = (float *)(nb + bv.cap);            // strain, staged: [nk][classes][kStrainOut]
  double *trace = (double *)(rows + (kStrain && bv.rows ? (bv.depth * sv.ncls * kStrainOut + 1) / 2 * 2 : 0));
  const BlockTile t = bv.tile[blockIdx.x];
  const int l = threadIdx.x;
  const int64_t N = p.ntot;
  // ---- what the time loop never changes: before the wait for the previous launch.  Topology, tiles
  // and parameters are written when a handle, a recording or a strain is set up, with the stream
  // idle.  The rows of strained elements (cdtf, gaxf, wdxf, kdxf and their columns of hpq) are
  // rewritten by strain_apply in the same chain: their values read here are not used, row_take(0)
  // and the re-read of gp and gd replace them after the wait.
  int dist = 1 << 20;
  int64_t j = -1;
  if (l < t.cnt) {
    j = t.s + l;
    dist = 0;
    nb[l] = make_ushort4(l > 0 ? l - 1 : l, l + 1 < t.cnt ? l + 1 : l, l, 0);
  } else if (l < t.cnt + t.nh) {
    const int4 h = bv.halo[t.h0 + l - t.cnt];
    j = h.x;
    dist = h.z >> 16;
    nb[l] = make_ushort4(h.y & 0xffff, (unsigned)h.y >> 16, h.z & 0xffff, 0);
  }
  uint32_t fl = F_TERM;
  uint32_t cls = 0;
  float cdt = 0, g0 = 0, wdx = 0, kdx = 0;
  HHParams32 q;
#pragma unroll
  for (int u = 0; u < 12; u++) q.v[u] = 0;
  int sc = -1;  // strain class
  if (j >= 0) {
    fl = p.eflags[j];
    cdt = p.cdtf[j];
    g0 = p.gaxf[j];
    if (p.hp_cls) cls = p.hp_cls[j];
    if (kStrain) sc = bv.scls[j] - 1;
    if (fl & F_HH) {
      if (kDense)
        q = hh_params32(p.hpq, p.hp_cls ? (int64_t)cls : (p.hp_inst ? (int64_t)(fl >> INST_SHIFT) : j));
    } else {
      wdx = p.wdxf[j];
      kdx = p.kdxf[j];
    }
    G[l] = g0;
    if (kStrain) G[bv.cap + l] = g0;
  }
  __syncthreads();
  for (int e = l; e < t.nx; e += blockDim.x) {  // owned elements with far neighbours
    const ushort4 x = bv.spec[t.x0 + e];
    nb[x.x] = make_ushort4(x.y, x.z, x.w, 0);
  }
  __syncthreads();
  int lm = 0, lr = 0, ll = 0;
  float gp = 0, gd = 0;
  if (j >= 0) {
    const ushort4 x = nb[l];
    lm = x.x;
    lr = x.y;
    ll = x.z;
    gp = G[lr];
    gd = G[ll];
  }
  chain_acquire();  // the previous launch of the time loop has finished
  chain_release();
  // ---- state
  const bool hh = (fl & F_HH) != 0, term = (fl & F_TERM) != 0;
  double V = 0;
  float f = 0, m = 0, h = 0, n = 0;
  int left = 0, on0 = 1, on1 = 0;
  if (j >= 0) {
    V = Vin[j];
    if (hh) {
      m = gin[j];
      h = gin[N + j];
      n = gin[2 * N + j];
    }
    const InstDev in = p.inst[fl >> INST_SHIFT];
    const int64_t i0 = in.base + k0;
    left = clip_int(in.iend - i0);
    on0 = clip_int(in.ion - i0);
    on1 = clip_int(in.ioff - i0);
    f = d2f(V);
    F[l] = f;
  }
  const float inp = j >= 0 && (fl & F_INP) ? p.inpf[j] : 0.0f;
  // recording: an element's potential after every step goes to the trace column of its first
  // probe in the tile's list
  const int np = kRec ? t.p1 - t.p0 : 0;
  int col = -1;
  for (int e = 0; e < np && col < 0; e++)
    if (bv.probe[t.p0 + e].x == l) col = e;
  // strain: the classes' rows of these steps as FP32, staged when they are few; a strained
  // element takes its row before each step
  if (kStrain && bv.rows) {
    const int count = nk * sv.ncls * kStrainOut;
    const double *src = sv.tab + (int64_t)k0 * sv.ncls * kStrainOut;
    for (int u = l; u < count; u += blockDim.x) rows[u] = d2f(src[u]);
    __syncthreads();
  }
  auto row_take = [&](int k) {
    if (!kStrain || sc < 0) return;
    const float *o = rows + (k * sv.ncls + sc) * kStrainOut;
    const double *og = sv.tab + ((int64_t)(k0 + k) * sv.ncls + sc) * kStrainOut;
    auto at = [&](int u) { return bv.rows ? o[u] : d2f(og[u]); };
    cdt = at(0);
    g0 = at(1);
    G[(k & 1) * bv.cap + l] = g0;
    if (hh) {
#pragma unroll
      for (int u = 0; u < HP_ROWS; u++) q.v[u] = at(2 + u);
    } else {
      wdx = at(2);
      kdx = at(3);
    }
  };
  row_take(0);
  __syncthreads();
  // ---- steps
  for (int k = 0; k < nk; k++) {
    const float *Fk = F + (k & 1) * bv.cap;
    if (dist < nk - k) {  // the value after this step still reaches an owned element
      if (k < left && !(term && !hh)) {
        if (kStrain) {
          gp = G[(k & 1) * bv.cap + lr];
          gd = G[(k & 1) * bv.cap + ll];
        }
        const float vf = term ? Fk[lm] : f;
        float wd = wdx, kd = kdx;
        if (hh) {
          if (!kDense && !(kStrain && sc >= 0))
            q = hh_params32(p.hpq, p.hp_cls ? (int64_t)cls
                                            : (p.hp_inst ? (int64_t)(fl >> INST_SHIFT) : j));
          const float dv = vf - q.v[HP_REST];
          const GateStep32 s =
              hh_step32(dv + q.v[HP_LSNA], dv + q.v[HP_LSK], m, h, n, q.v[HP_DTMS], q.v[HP_GNA],
                        q.v[HP_GK], q.v[HP_GL], q.v[HP_ENA], q.v[HP_EK], q.v[HP_EL]);
          m = s.m;
          h = s.h;
          n = s.n;
          wd = s.W * q.v[HP_DX];
          kd = s.K * q.v[HP_DX];
        }
        if (!term) {
          float acc = 0.0f;
          if ((fl & F_BRANCH) && !(fl & F_DL_TERM)) acc = (Fk[ll] - vf) * gd;
          if (!(fl & F_DR_TERM)) acc = fmaf(Fk[lr] - vf, gp, acc);
          if (!(fl & F_MO_TERM)) acc = fmaf(Fk[lm] - vf, g0, acc);
          acc = fmaf(wd, vf, acc) + kd;
          if ((fl & F_INP) && k >= on0 && k <= on1) acc += inp;
          V = V + f2d(cdt * acc);
          f = d2f(V);
        }
      }
      F[((k + 1) & 1) * bv.cap + l] = f;
      if (kRec && col >= 0) trace[k * np + col] = V;
    }
    if (k + 1 < nk) row_take(k + 1);
    __syncthreads();
  }
  // ---- owned state out
  if (dist == 0) {
    if (!term || left <= 0) {
      Vout[j] = V;
      Fout[j] = f;
    }
    if (hh) {
      gout[j] = m;
      gout[N + j] = h;
      gout[2 * N + j] = n;
    }
  }
  if (kRec) record_tile(p, bv, t, r, k0, nk, trace, np);
}

// The FP64 form (no strain).  kLanes = 8: eight lanes per local element (hh_group_step); 1: one
// thread each.  What bounds it is the FP64 pipe: a warp's dependent operations take 64 cycles
// each, about 39 in sequence per step on eight lanes and 115 on one, and independent warps of an
// SM partition share it.  So a small axon spreads over all SMs, four warps each, 16 local
// elements of which half are halo at 4 steps per launch.
template <int kLanes, bool kRec>
__global__ void __launch_bounds__(256, 2)
    explicit_block_f64(PackView p, BlockView bv, int k0, int nk, const double *Vin, double *Vout,
                       const double *gin, double *gout, RecView r) {
  extern __shared__ __align__(16) unsigned char bsm[];
  double *Vs = (double *)bsm;                    // [2][cap]
  double *G = Vs + 2 * bv.cap;                   // [cap]
  double *trace = G + bv.cap;                    // [nk][probes]
  ushort4 *nb = (ushort4 *)(trace + bv.depth * bv.max_probes);
  const BlockTile t = bv.tile[blockIdx.x];
  const int l = threadIdx.x / kLanes, q = threadIdx.x % kLanes;
  const int64_t N = p.ntot;
  exp64_prefetch();
  // ---- what the time loop never changes: before the wait for the previous launch (topology and
  // conductances; FP64 packs with a strain, which rewrites conductances, do not come here)
  int dist = 1 << 20;
  int64_t j = -1;
  if (l < t.cnt) {
    j = t.s + l;
    dist = 0;
    if (q == 0) nb[l] = make_ushort4(l > 0 ? l - 1 : l, l + 1 < t.cnt ? l + 1 : l, l, 0);
  } else if (l < t.cnt + t.nh) {
    const int4 h = bv.halo[t.h0 + l - t.cnt];
    j = h.x;
    dist = h.z >> 16;
    if (q == 0) nb[l] = make_ushort4(h.y & 0xffff, (unsigned)h.y >> 16, h.z & 0xffff, 0);
  }
  uint32_t fl = F_TERM;
  double g0 = 0;
  if (j >= 0) {
    fl = p.topo[j].flags;
    g0 = p.gax[j];
    if (q == 0) G[l] = g0;
  }
  const bool hh = (fl & F_HH) != 0, term = (fl & F_TERM) != 0;
  const bool dl = (fl & F_BRANCH) && !(fl & F_DL_TERM), dr = !(fl & F_DR_TERM), mo = !(fl & F_MO_TERM);
  __syncthreads();
  for (int e = threadIdx.x; e < t.nx; e += blockDim.x) {  // owned elements with far neighbours
    const ushort4 x = bv.spec[t.x0 + e];
    nb[x.x] = make_ushort4(x.y, x.z, x.w, 0);
  }
  __syncthreads();
  int lm = 0, lr = 0, ll = 0;
  double gdr = 0, gdl = 0;
  if (j >= 0) {
    const ushort4 x = nb[l];
    lm = x.x;
    lr = x.y;
    ll = x.z;
    gdr = G[lr];
    gdl = G[ll];
  }
  chain_acquire();  // the previous launch of the time loop has finished
  chain_release();
  // ---- state
  double V = 0, gate = 0, h0 = 0, n0 = 0;  // kLanes = 8: gate is lane 0's m, 2's h, 4's n
  double cdt = 0, wdx = 0, kdx = 0, inp = 0;
  int left = 0, on0 = 1, on1 = 0;
  HHGroup hg{};
  double lsk = 0, gk = 0, ek = 0;  // kLanes = 1: the K side (hg holds the Na side)
  if (kLanes == 8) hg.r = hh_lane(q < 6 ? q : 5);
  if (j >= 0) {
    V = Vin[j];
    if (q == 0) Vs[l] = V;
    const InstDev in = p.inst[fl >> INST_SHIFT];
    const int64_t i0 = in.base + k0;
    left = clip_int(in.iend - i0);
    on0 = clip_int(in.ion - i0);
    on1 = clip_int(in.ioff - i0);
    cdt = p.cdt[j];
    if (hh) {
      const int64_t L = p.hp_ld;
      const double *hp = p.hp + hp_col(p, j, fl >> INST_SHIFT);
      const bool na = kLanes == 1 || q < 4;
      hg.ls = hp[(na ? HP_LSNA : HP_LSK) * L];
      hg.rest = hp[HP_REST * L];
      hg.dt = hp[HP_DTMS * L];
      hg.g = hp[(na ? HP_GNA : HP_GK) * L];
      hg.GL = hp[HP_GL * L];
      hg.e = hp[(na ? HP_ENA : HP_EK) * L];
      hg.EL = hp[HP_EL * L];
      hg.dx = hp[HP_DX * L];
      if (kLanes == 1) {
        lsk = hp[HP_LSK * L];
        gk = hp[HP_GK * L];
        ek = hp[HP_EK * L];
        gate = gin[j];
        h0 = gin[N + j];
        n0 = gin[2 * N + j];
      } else if (q == 0 || q == 2 || q == 4) {
        gate = gin[(q >> 1) * N + j];
      }
    } else {
      wdx = p.wdx[j];
      kdx = p.kdx[j];
    }
    if (fl & F_INP) inp = p.inp[j];
  }
  const int np = kRec ? t.p1 - t.p0 : 0;
  int col = -1;  // the trace column (see explicit_block_mixed)
  for (int e = 0; e < np && col < 0; e++)
    if (bv.probe[t.p0 + e].x == l) col = e;
  __syncthreads();
  // ---- steps
  for (int k = 0; k < nk; k++) {
    const double *Vk = Vs + (k & 1) * bv.cap;
    const bool reach = dist < nk - k;  // the value after this step still reaches an owned element
    const bool act = reach && k < left && !(term && !hh);
    double dd[3] = {0, 0, 0}, wd = wdx, kd = kdx;
    const double v = j >= 0 ? (term ? Vk[lm] : (kLanes == 1 ? V : Vk[l])) : 0.0;
    if (kLanes == 8) {
      const int at = q == 1 ? lr : q == 3 ? lm : q == 5 ? ll : l;
      double g2 = gate, kg;
      const double wg = hh_group_step(q, hg, v, j >= 0 ? Vk[at] : 0.0, g2, kg, dd);
      if (hh) {
        if (act) gate = g2;
        wd = wg;
        kd = kg;
      }
    } else if (act) {
      dd[0] = Vk[lr] - v;
      dd[1] = Vk[lm] - v;
      dd[2] = Vk[ll] - v;
      if (hh) {
        const GateStep64 s = hh_step64(v, gate, h0, n0, hg.ls, lsk, hg.rest, hg.dt, hg.g, gk, hg.GL,
                                       hg.e, ek, hg.EL);
        gate = s.m;
        h0 = s.h;
        n0 = s.n;
        wd = s.W * hg.dx;
        kd = s.K * hg.dx;
      }
    }
    if (q == 0 && reach) {
      if (act && !term) {
        const bool on = (fl & F_INP) && k >= on0 && k <= on1;
        V = f64_update(v, dl, dd[2], gdl, dr, dd[0], gdr, mo, dd[1], g0, wd, kd, on, inp, cdt);
      }
      Vs[((k + 1) & 1) * bv.cap + l] = V;
      if (kRec && col >= 0) trace[k * np + col] = V;
    }
    __syncthreads();
  }
  // ---- owned state out
  if (dist == 0) {
    if (q == 0 && (!term || left <= 0)) Vout[j] = V;
    if (hh) {
      if (kLanes == 1) {
        gout[j] = gate;
        gout[N + j] = h0;
        gout[2 * N + j] = n0;
      } else if (q == 0 || q == 2 || q == 4) {
        gout[(q >> 1) * N + j] = gate;
      }
    }
  }
  if (kRec) record_tile(p, bv, t, r, k0, nk, trace, np);
}

size_t block_smem(const BlockView &bv, const StrainView &s) {
  const bool strain = s.n > 0;
  return (size_t)bv.cap * (8 + (strain ? 8 : 4) + 8) +
         (strain && bv.rows ? 4 * (size_t)bv.depth * s.ncls * kStrainOut : 0) +
         8 * (size_t)bv.depth * bv.max_probes + 8;
}

}  // namespace

// Depth and tile size.  A halo costs about 2.5 elements per step of depth (two ends of the
// range and some branches; more on bushy trees of short branches), a launch boundary about 4 us.
// Packs that fit the SMs at once (1024 resident threads per SM dense, 1536 sparse) are
// launch-bound, so they take 8 or 16 steps and the tile size that loads the fullest SM least;
// larger ones stream: 8 steps hide the traffic (60 B per launch) and the loads' instructions
// behind the arithmetic, and large tiles keep the halo small.  Whatever the plan then turns out
// to hold decides (block_cost).
static void block_shape(const PackView &pv, int &depth, int &cap) {
  const bool dense = pv.hh_dense != 0;
  const int sms = pv.sms > 0 ? pv.sms : 1;
  const int64_t N = pv.ntot, resident = (int64_t)sms * (dense ? 1024 : 1536);
  depth = N <= resident && !dense ? 16 : 8;
  const int largest = dense ? 512 : 256;
  cap = largest;
  if (N > resident) return;
  int64_t best = -1;
  for (int c = 64; c <= largest; c *= 2) {
    const int own = c - 5 * depth / 2;
    if (own < c / 3) continue;
    const int64_t tiles = (N + own - 1) / own, load = (tiles + sms - 1) / sms * c;
    if (best < 0 || load < best) {
      best = load;
      cap = c;
    }
  }
}

static bool build_block_plan(const HostPack &host, int depth, int cap, BlockPlan &plan);
static unsigned plan_threads(int64_t N);

// Estimated microseconds per step of a plan, and of the per-step kernels: a launch boundary and
// the elements' share (measured on 5.4 and 22 million compartments: 9 to 11 ps per local
// element, 14.5 ps per element one step at a time; small packs 4.6 us per launch).
static double block_cost(const BlockPlan &P) {
  double local = 0;
  for (const BlockTile &t : P.tile) local += t.cnt + t.nh;
  return 4.0 / P.depth + 1e-5 * local;
}

// FP64 shapes, by estimated microseconds per step: a launch boundary of 3 us, 1.3 us per round of
// 16 eight-lane elements on an SM and 3.8 us per round of 128 one-thread ones (39 and 115
// operations of 64 cycles), against the per-step kernels' 3.3 us and the same rounds without
// halos.  Above a million elements the launch boundary is nothing to the rounds.
struct F64Shape {
  int lanes, depth, cap;
};
constexpr F64Shape kF64Shapes[] = {{8, 4, 16}, {8, 4, 32}, {1, 8, 128}, {1, 4, 128}, {1, 4, 256}, {1, 2, 256}};
constexpr int64_t kF64MaxElems = 1000000;

static double f64_rounds(int64_t local, int lanes, int64_t sms) {
  const double per = lanes == 8 ? 16.0 : 128.0, x = (double)local / (double)sms / per;
  return (lanes == 8 ? 1.3 : 3.8) * (x < 4 ? std::max(1.0, std::ceil(x - 0.05)) : x);
}
static double f64_single_cost(int64_t N, const PackView &pv) {
  const int64_t sms = pv.sms > 0 ? pv.sms : 1;
  return 3.3 + std::min(f64_rounds(N, 1, sms), N <= 8192 ? f64_rounds(N, 8, sms) : 1e30);
}
static double f64_cost(const F64Shape &s, int64_t tiles, const PackView &pv) {
  const int64_t sms = pv.sms > 0 ? pv.sms : 1;
  // whole tiles go to an SM, so the fullest SM holds ceil(tiles / SMs) of them
  return 3.0 / s.depth + f64_rounds((tiles + sms - 1) / sms * s.cap * sms, s.lanes, sms);
}

static bool choose_f64(const HostPack &host, const PackView &pv, BlockPlan &plan) {
  const int64_t N = host.ntot;
  if (N > kF64MaxElems) return false;
  double best = f64_single_cost(N, pv);
  bool found = false;
  for (const F64Shape &s : kF64Shapes) {
    const int own = s.cap - 2 * s.depth;  // at best: a cable
    if (f64_cost(s, (N + own - 1) / own, pv) >= best) continue;
    BlockPlan P;
    if (!build_block_plan(host, s.depth, s.cap, P)) continue;
    const double cost = f64_cost(s, (int64_t)P.tile.size(), pv);
    if (cost >= best) continue;
    best = cost;
    P.lanes = s.lanes;
    plan = std::move(P);
    found = true;
  }
  return found;
}

bool choose_block_plan(const HostPack &host, const PackView &pv, bool mixed, BlockPlan &plan) {
  if (!mixed) return choose_f64(host, pv, plan);
  int depth = 0, cap = 0;
  block_shape(pv, depth, cap);
  const int largest = pv.hh_dense ? 512 : 256;
  double best = 4.6 + 1.45e-5 * (double)host.ntot;
  bool found = false;
  for (int d = depth, c = cap; d >= 2;) {
    BlockPlan P;
    const bool ok = build_block_plan(host, d, c, P);
    const double cost = ok ? block_cost(P) : 0.0;
    if (ok && cost < best) {
      best = cost;
      plan = std::move(P);
      found = true;
    }
    // good as it is: the halos are below a third
    if (ok && cost < 4.0 / d + 1.33e-5 * (double)host.ntot) break;
    if (c < largest)
      c = largest;
    else
      d /= 2;
  }
  return found;
}

// Whether `steps` steps are worth a plan: what they would save, against the plan's making.  Both are
// estimates from what was measured (16 host cores, a first call on a fresh handle):
//  - making: 60 us, up to 150 for allocations and copies, 55 us per further host thread, and over the
//    threads (16 of them at most: a container's share of the cores can be less than the system says)
//    0.25 us for each terminal (the elements around a branch are searched again for every tile) and
//    3.5 ns for each element; and 0.2 ns per element for the upload: 0.12 ms for a 10,000-element tree,
//    0.7 ms for 24 bushy trees (102,815 elements, 4,400 terminals), 0.6 ms for a myelinated axon of
//    199,202, 1.5 ms for a million elements, 13 ms for 1024 trees (22 million);
//  - saved per step, mixed: 4.3 us per launch, or 2.5 and 14.5 ps per element if that is more, becomes
//    2 us per depth and 6.8 ps per local element (102,815 elements 4.5 -> 1.2 us, a million 18.3 -> 7.9);
//    FP64: half of what choose_f64's estimates say (a 1 cm axon 3.7 -> 2.7 us, 10,000 elements 6.8 ->
//    5.4).
// With 128 steps for every pack, the 24 trees' first call of 128 steps took 1.28 ms instead of 0.82.
bool block_plan_pays(const HostPack &host, const PackView &pv, bool mixed, int64_t steps) {
  const double N = (double)host.ntot;
  const double threads = plan_threads(host.ntot);
  const double making = 60.0 + std::min(150.0, 0.0015 * N) + 55.0 * (threads - 1) + 0.0002 * N +
                        (0.25 * (double)host.terms.size() + 0.0035 * N) / std::min(threads, 16.0);
  double saved;
  if (mixed) {
    int depth = 0, cap = 0;
    block_shape(pv, depth, cap);
    saved = std::max(4.3, 2.5 + 1.45e-5 * N) - (2.0 / depth + 6.8e-6 * 1.15 * N);
  } else {
    double best = f64_single_cost(host.ntot, pv);
    const double single = best;
    for (const F64Shape &s : kF64Shapes) {
      const int64_t own = s.cap - 2 * s.depth;
      best = std::min(best, f64_cost(s, (host.ntot + own - 1) / own, pv));
    }
    saved = host.ntot > kF64MaxElems ? 0.0 : 0.5 * (single - best);
  }
  return saved > 0 && (double)steps * saved >= making;
}

// Host threads of a plan.  A thread's start and its first allocations take about 55 us in a process
// of many libraries, so small packs take four (a myelinated axon of 199,202 elements: 0.68 ms on
// one, 0.42 on four, 0.83 to 1.4 on thirteen; 24 bushy trees 1.2, 0.6 and 0.8).
static unsigned plan_threads(int64_t N) {
  const int64_t chunks = (N + (1 << 14) - 1) / (1 << 14);
  return (unsigned)std::min<int64_t>({chunks, std::max<int64_t>(4, N >> 17), (int64_t)host_threads()});
}

// The plan of elements [c0, c1) (local entries h0, x0 count from P's own lists); false when some
// tile would hold fewer than a quarter of its elements itself (a dense tangle of branches).
static bool tile_range(const HostPack &host, int depth, int cap, int64_t c0, int64_t c1, BlockPlan &P) {
  struct H {
    int64_t g;
    int dist;
  };
  // what element j's step reads besides its own state, -1 where it reads nothing
  auto deps = [&](int64_t j, int64_t (&d)[3]) {
    const Topo &t = host.topo[j];
    d[0] = d[1] = d[2] = -1;
    if (t.flags & F_TERM) {
      if (t.flags & F_HH) d[0] = (t.flags & F_ROOT) ? j + 1 : (int64_t)t.mother;
      return;
    }
    if (!(t.flags & F_MO_TERM)) d[0] = t.mother;
    if (!(t.flags & F_DR_TERM)) d[1] = t.dr;
    if ((t.flags & F_BRANCH) && !(t.flags & F_DL_TERM)) d[2] = t.dl;
  };
  // the elements with a neighbour that is not j - 1 or j + 1: with the two ends of a tile the only
  // ones whose step can read outside it
  std::vector<int64_t> far;
  for (int64_t j = c0; j < c1; j++)
    if (host.topo[j].flags & F_XTOPO) far.push_back(j);
  std::vector<H> halo;
  std::vector<int64_t> key(4096, -1);  // open-addressing map: element -> local index
  std::vector<int> val(4096);
  std::vector<size_t> used;
  auto slot = [&](int64_t g) {
    size_t h = (size_t)(g * 0x9E3779B97F4A7C15ull >> 40) & 4095;
    while (key[h] >= 0 && key[h] != g) h = (h + 1) & 4095;
    return h;
  };
  int64_t s = c0;
  size_t f0 = 0;                   // the first of `far` at or after s
  int64_t want = cap - 2 * depth;  // then what the last tile held and a little more
  while (s < c1) {
    int64_t cnt = std::min(want, c1 - s);
    int64_t d[3];
    // f(j) for the tile's elements that may read outside it, in ascending order
    auto each = [&](auto f) {
      size_t q = f0;
      if (q == far.size() || far[q] != s) f(s);
      for (; q < far.size() && far[q] < s + cnt; q++) f(far[q]);
      if (cnt > 1 && (q == f0 || far[q - 1] != s + cnt - 1)) f(s + cnt - 1);
    };
    for (bool fits = false; !fits;) {
      for (size_t q : used) key[q] = -1;
      used.clear();
      halo.clear();
      bool full = false;
      auto add = [&](int64_t g, int dist) {
        if (g < 0 || (g >= s && g < s + cnt)) return;
        const size_t h = slot(g);
        if (key[h] == g) return;
        if (cnt + (int64_t)halo.size() >= cap) {
          full = true;
          return;
        }
        key[h] = g;
        used.push_back(h);
        val[h] = (int)(cnt + (int64_t)halo.size());
        halo.push_back(H{g, dist});
      };
      each([&](int64_t j) {
        if (full) return;
        deps(j, d);
        for (int64_t g : d) add(g, 1);
      });
      for (size_t q = 0; q < halo.size() && !full; q++) {
        if (halo[q].dist >= depth) break;  // sorted by distance
        deps(halo[q].g, d);
        for (int64_t g : d) add(g, halo[q].dist + 1);
      }
      fits = !full;
      if (!fits) {
        cnt -= std::max<int64_t>(depth, cnt / 16);
        if (cnt < std::max(1, cap / 4)) return false;
      }
    }
    auto local = [&](int64_t g, int self) -> int {
      if (g < 0) return self;
      if (g >= s && g < s + cnt) return (int)(g - s);
      const size_t h = slot(g);
      return key[h] == g ? val[h] : self;
    };
    BlockTile t{};
    t.s = (int32_t)s;
    t.cnt = (int32_t)cnt;
    t.nh = (int32_t)halo.size();
    t.h0 = (int32_t)P.halo.size();
    t.x0 = (int32_t)P.spec.size();
    each([&](int64_t j) {
      const int l = (int)(j - s);
      deps(j, d);
      P.spec.push_back(make_ushort4((unsigned short)l, (unsigned short)local(d[0], l),
                                    (unsigned short)local(d[1], l), (unsigned short)local(d[2], l)));
    });
    t.nx = (int32_t)P.spec.size() - t.x0;
    for (size_t q = 0; q < halo.size(); q++) {
      const int l = (int)(cnt + (int64_t)q);
      int nbr[3] = {l, l, l};
      if (halo[q].dist < depth) {
        deps(halo[q].g, d);
        for (int u = 0; u < 3; u++) nbr[u] = local(d[u], l);
      }
      P.halo.push_back(make_int4((int)halo[q].g, nbr[0] | (nbr[1] << 16), nbr[2] | (halo[q].dist << 16), 0));
    }
    P.tile.push_back(t);
    s += cnt;
    while (f0 < far.size() && far[f0] < s) f0++;
    want = std::min<int64_t>(cap - 2 * depth, cnt + std::max(depth, cap / 32));
  }
  return true;
}

// Tiles of at most `cap` local elements for `depth` steps per launch; false where tile_range says
// so.  Ranges of elements are tiled by one host thread each.
static bool build_block_plan(const HostPack &host, int depth, int cap, BlockPlan &plan) {
  plan.depth = depth;
  plan.cap = cap;
  const int64_t N = host.ntot, chunk = std::min<int64_t>(1 << 16, std::max<int64_t>(1 << 14, N / 64));
  const int64_t nc = (N + chunk - 1) / chunk;
  std::vector<BlockPlan> part(nc);
  std::atomic<bool> tangle(false);
  parallel_for(nc, [&](int64_t c) {
    if (tangle) return;
    if (!tile_range(host, depth, cap, c * chunk, std::min(N, (c + 1) * chunk), part[c])) tangle = true;
  }, plan_threads(N));
  if (tangle) return false;
  size_t nt = 0, nh = 0, nx = 0;
  for (int64_t c = 0; c < nc; c++) {
    nt += part[c].tile.size();
    nh += part[c].halo.size();
    nx += part[c].spec.size();
  }
  if (nh >= ((size_t)1 << 31) || nx >= ((size_t)1 << 31)) return false;
  plan.tile.reserve(nt);
  plan.halo.reserve(nh);
  plan.spec.reserve(nx);
  for (int64_t c = 0; c < nc; c++) {
    for (BlockTile t : part[c].tile) {
      t.h0 += (int32_t)plan.halo.size();
      t.x0 += (int32_t)plan.spec.size();
      plan.tile.push_back(t);
    }
    plan.halo.insert(plan.halo.end(), part[c].halo.begin(), part[c].halo.end());
    plan.spec.insert(plan.spec.end(), part[c].spec.begin(), part[c].spec.end());
  }
  return true;
}

int launch_explicit_block(const PackView &pv, const BlockView &bv, int precision, int k0, int nk,
                          const double *Vin, double *Vout, float *Fout, const void *gin, void *gout,
                          const RecView &r, const StrainView &s, cudaStream_t st) {
  if (nk < 1 || nk > bv.depth) return NRT_EINVAL;
  const bool rec = r.nprobe > 0 && bv.max_probes > 0;
  if (precision != NRT_MIXED) {
    auto kern = bv.lanes == 8 ? (rec ? explicit_block_f64<8, true> : explicit_block_f64<8, false>)
                              : (rec ? explicit_block_f64<1, true> : explicit_block_f64<1, false>);
    const size_t smem = (size_t)bv.cap * (24 + 8) + 8 * (size_t)bv.depth * bv.max_probes;
    NRT_CUDA(launch_chained(kern, bv.ntiles, bv.cap * bv.lanes, smem, st, pv, bv, k0, nk, Vin, Vout,
                            (const double *)gin, (double *)gout, r));
    return NRT_OK;
  }
  const bool strain = s.n > 0;
  auto pick = [&](auto with_rec) {
    constexpr bool R = decltype(with_rec)::value;
    return pv.hh_dense ? (strain ? explicit_block_mixed<true, true, R> : explicit_block_mixed<true, false, R>)
                       : (strain ? explicit_block_mixed<false, true, R> : explicit_block_mixed<false, false, R>);
  };
  auto kern = rec ? pick(std::true_type()) : pick(std::false_type());
  NRT_CUDA(launch_chained(kern, bv.ntiles, bv.cap, block_smem(bv, s), st, pv, bv, k0, nk, Vin, Vout,
                          Fout, (const float *)gin, (float *)gout, r, s));
  return NRT_OK;
}

}  // namespace nrt
