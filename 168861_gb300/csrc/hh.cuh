// Hodgkin-Huxley rate functions and the forward-Euler gate step, FP64 and FP32 forms.
//
// Model: src/coupling.cpp:25-48 (hhRate_Const), gate and conductance update
// src/solverEx-cpu.cpp:106-127, W and K src/discretization.cpp:99-104.  Voltages enter in
// mV relative to rest (SCALE 0.001, inc/configuration.h:36) and dt in ms.
#pragma once
#include <cuda_runtime.h>

#include "math64.cuh"

namespace nrt {

struct GateStep64 {
  double m, h, n;   // gates after the step
  double W, K;      // membrane coefficients with the new gates
};

// The six FP64 rates (order: alpha_m, beta_m, alpha_h, beta_h, alpha_n, beta_n) are
// each one exponential and one quotient or product of it, of the potential v that the rate
// reads (v_Na for the first four, v_K for the others).  hh_rate64 gives rate q with the same
// operations for every q -- so lanes of a warp can evaluate different rates of one element
// without diverging (HHLane holds a lane's constants) -- and with the value of the reference's
// expression:
//   alpha_m = xm / (e^xm - 1),            xm = 2.5 - 0.1 v_Na
//   beta_m  = 4 e^(-v_Na/18)              alpha_h = 0.07 e^(-v_Na/20)
//   beta_h  = 1 / (e^(3 - 0.1 v_Na) + 1)
//   alpha_n = (0.1 - 0.01 v_K) / (e^xn - 1),  xn = 1 - 0.1 v_K
//   beta_n  = 0.125 e^(-v_K/80)
// (the factors 4 and 0.125 go into the exponential's scale, which is exact).  The a - b c terms
// are explicit fused multiply-adds, so that a constant q and a q chosen per lane round alike.
struct HHLane {
  double a, b;    // the exponent, a v + b
  double c, k;    // e + c under the quotient; k e without one
  int scale;
  bool quot;
};
__device__ __forceinline__ HHLane hh_lane(int q) {
  HHLane r;
  r.a = q == 1 ? -1.0 / 18.0 : q == 2 ? -1.0 / 20.0 : q == 5 ? -1.0 / 80.0 : -0.1;
  r.b = q == 0 ? 2.5 : q == 3 ? 3.0 : q == 4 ? 1.0 : 0.0;
  r.c = q == 3 ? 1.0 : -1.0;
  r.k = q == 2 ? 0.07 : 1.0;
  r.scale = q == 1 ? 2 : q == 5 ? -3 : 0;
  r.quot = q == 0 || q == 3 || q == 4;
  return r;
}
__device__ __forceinline__ double hh_rate64(int q, const HHLane &r, double v) {
  const double x = r.b == 0.0 ? v * r.a : fma(r.a, v, r.b);
  const double e = exp64(x, r.scale);
  if (!r.quot) return r.k == 1.0 ? e : r.k * e;
  return div64(q == 0 ? x : q == 3 ? 1.0 : fma(-0.01, v, 0.1), e + r.c);
}
// The same without branches, for lanes that evaluate different rates.
__device__ __forceinline__ double hh_rate64_lane(int q, const HHLane &r, double v) {
  const double x = fma(r.a, v, r.b);  // b = 0: the product, rounded once
  const double e = exp64(x, r.scale);
  const double n4 = fma(-0.01, v, 0.1);
  const double num = !r.quot ? 1.0 : q == 0 ? x : q == 3 ? 1.0 : n4;
  const double d = div64(num, r.quot ? e + r.c : 1.0);
  const double ke = r.k * e;
  return r.quot ? d : ke;
}

// The forward-Euler gate step and W, K from the six rates.  The fused multiply-adds are
// written out: a - b c + d e style sums have two ways to fuse, and left to the compiler the
// choice could differ between kernels that inline this (the lanes kernel and the others
// must agree bit for bit).
__device__ __forceinline__ GateStep64 hh_gates64(double am, double bm, double ah, double bh,
                                                 double an, double bn, double m0, double h0,
                                                 double n0, double dt_ms, double gNa,
                                                 double gK, double GL, double ENa, double EK,
                                                 double EL) {
  GateStep64 r;
  r.m = fma(dt_ms, fma(am, 1.0 - m0, -(bm * m0)), m0);
  r.h = fma(dt_ms, fma(ah, 1.0 - h0, -(bh * h0)), h0);
  r.n = fma(dt_ms, fma(an, 1.0 - n0, -(bn * n0)), n0);
  const double G_Na = gNa * r.m * r.m * r.m * r.h;
  const double G_K = gK * r.n * r.n * r.n * r.n;
  r.W = -(G_Na + G_K + GL);
  r.K = fma(GL, EL, fma(G_K, EK, G_Na * ENa));
  return r;
}

// FP64: the reference's expressions with constant divisions turned into products.
__device__ __forceinline__ GateStep64 hh_step64(double v, double m0, double h0, double n0,
                                                double ls_na, double ls_k, double rest,
                                                double dt_ms, double gNa, double gK, double GL,
                                                double ENa, double EK, double EL) {
  const double vna = ((v + ls_na) - rest) * 1000.0;
  const double vk = ((v + ls_k) - rest) * 1000.0;
  return hh_gates64(hh_rate64(0, hh_lane(0), vna), hh_rate64(1, hh_lane(1), vna),
                    hh_rate64(2, hh_lane(2), vna), hh_rate64(3, hh_lane(3), vna),
                    hh_rate64(4, hh_lane(4), vk), hh_rate64(5, hh_lane(5), vk), m0,
                    h0, n0, dt_ms, gNa, gK, GL, ENa, EK, EL);
}

// The explicit update V' = v + dT/(c_m dX) (fluxes + W dX v + K dX + I) with the reference's
// order of summation (src/solverEx-cpu.cpp:141-152); d*: potential differences to DL, DR and
// mother, g*: their conductances.  Written out in fused multiply-adds so that every FP64 kernel
// rounds alike.
__device__ __forceinline__ double f64_update(double v, bool has_dl, double ddl, double gdl,
                                             bool has_dr, double ddr, double gdr, bool has_mo,
                                             double dmo, double gmo, double wdx, double kdx,
                                             bool on, double inp, double cdt) {
  double acc = has_dl ? ddl * gdl : 0.0;
  if (has_dr) acc = fma(ddr, gdr, acc);
  if (has_mo) acc = fma(dmo, gmo, acc);
  acc = fma(wdx, v, acc);
  acc = acc + kdx;
  if (on) acc = acc + inp;  // adding a zero input is exact
  return fma(cdt, acc, v);
}

// One FP64 compartment-step on a group of eight lanes (q: lane in the group; every lane of the
// warp takes part).  A dependent FP64 operation costs a warp 64 cycles, so what counts is the
// number of operations in sequence: about 39 here, 115 in one thread.  Lanes 0-5 evaluate a
// rate each; the gates live in lanes 0 (m), 2 (h) and 4 (n) and move together; G_Na and W go
// through lane 0, G_K and K through lane 4, by the same operations on different operands;
// lanes 1, 3 and 5 form the potential differences.  Lane 0 returns W dX, kdx its K dX and d the
// differences.  The same values as hh_step64 and f64_update, bit for bit.
struct HHGroup {
  HHLane r;
  double ls, rest, dt, g, GL, e, EL, dx;  // ls of the lane's rate; g, e: Na in lanes 0-3, else K
};
__device__ __forceinline__ double hh_group_step(int q, const HHGroup &p, double v, double vn,
                                                double &gate, double &kdx, double (&d)[3]) {
  constexpr unsigned all = 0xffffffffu;
  const double diff = vn - v;  // lanes 1, 3, 5: DR, mother, DL
  const double rate = hh_rate64_lane(q, p.r, ((v + p.ls) - p.rest) * 1000.0);
  d[0] = __shfl_sync(all, diff, 1, 8);
  d[1] = __shfl_sync(all, diff, 3, 8);
  d[2] = __shfl_sync(all, diff, 5, 8);
  const double beta = __shfl_down_sync(all, rate, 1, 8);
  gate = fma(p.dt, fma(rate, 1.0 - gate, -(beta * gate)), gate);
  const double h = __shfl_sync(all, gate, 2, 8);
  double G = p.g * gate * gate * gate;  // lane 0: g_Na m^3 h, lane 4: g_K n^4
  G = G * (q < 4 ? h : gate);
  const double Go = __shfl_xor_sync(all, G, 4, 8);
  // lane 0: (G_Na + G_K) + G_L; lane 4: G_Na E_Na, + G_K E_K, + G_L E_L
  const double ena = __shfl_xor_sync(all, p.e, 4, 8);
  const bool na = q < 4;
  const double t1 = fma(na ? G : Go, na ? 1.0 : ena, na ? Go : 0.0);
  const double t2 = fma(na ? p.GL : G, na ? 1.0 : p.e, t1);
  const double t3 = fma(p.GL, p.EL, t2);
  const double w = (na ? -t2 : t3) * p.dx;
  kdx = __shfl_sync(all, w, 4, 8);
  return w;
}

// e^x and a / b by the fast units in their flush-to-zero forms: the values of __expf and
// __fdividef wherever neither the result nor b is subnormal (rates below 1e-38 per ms), without
// the scaling code around them (3 instructions less each, of about 260 per compartment-step).
__device__ __forceinline__ float fast_exp(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}
__device__ __forceinline__ float fast_div(float a, float b) {
  float y;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}

// x / (e^x - 1), the shape of alpha_m and alpha_n, with its removable singularity at 0
// handled by the series 1 / (1 + x/2 + x^2/6) for |x| < 1e-3.  Both branches use the fast
// reciprocal (a relative error of a few 1e-7, far below the FP32 gates' own rounding).
__device__ __forceinline__ float xexpm1_ratio(float x, float ex) {
  const float den = fabsf(x) < 1e-3f ? fmaf(x, fmaf(x, 1.0f / 6.0f, 0.5f), 1.0f) : ex - 1.0f;
  const float num = fabsf(x) < 1e-3f ? 1.0f : x;
  return fast_div(num, den);
}

struct GateStep32 {
  float m, h, n, W, K;
};

// FP32 form for the mixed-precision path.  dv_na / dv_k are (V + LS - rest) in volts,
// formed in FP64 by the caller and rounded once.  exp(3 - 0.1 v) is e^0.5 * exp(2.5 - 0.1 v).
__device__ __forceinline__ GateStep32 hh_step32(float dv_na, float dv_k, float m0, float h0,
                                                float n0, float dt_ms, float gNa, float gK,
                                                float GL, float ENa, float EK, float EL) {
  const float vna = dv_na * 1000.0f;
  const float vk = dv_k * 1000.0f;
  const float xm = fmaf(-0.1f, vna, 2.5f);
  const float exm = fast_exp(xm);
  const float am = xexpm1_ratio(xm, exm);
  const float bm = 4.0f * fast_exp(vna * (-1.0f / 18.0f));
  const float ah = 0.07f * fast_exp(vna * (-1.0f / 20.0f));
  const float bh = fast_div(1.0f, fmaf(exm, 1.6487212707001282f, 1.0f));
  const float xn = fmaf(-0.1f, vk, 1.0f);
  const float an = 0.1f * xexpm1_ratio(xn, fast_exp(xn));
  const float bn = 0.125f * fast_exp(vk * (-1.0f / 80.0f));
  GateStep32 r;
  r.m = fmaf(dt_ms, am * (1.0f - m0) - bm * m0, m0);
  r.h = fmaf(dt_ms, ah * (1.0f - h0) - bh * h0, h0);
  r.n = fmaf(dt_ms, an * (1.0f - n0) - bn * n0, n0);
  const float G_Na = gNa * r.m * r.m * r.m * r.h;
  const float n2 = r.n * r.n;
  const float G_K = gK * n2 * n2;
  r.W = -(G_Na + G_K + GL);
  r.K = fmaf(G_Na, ENa, fmaf(G_K, EK, GL * EL));
  return r;
}

}  // namespace nrt
