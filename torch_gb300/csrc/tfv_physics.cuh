// Device physics of TORCH's Cartesian finite-volume step, templated on the
// arithmetic type R.
//
// double — the reference-faithful path.  Every expression keeps the operation
//   order of the NumPy reference so that, compiled without FMA contraction
//   (-fmad=false), it reproduces the reference bit for bit: `a * b * c` in
//   Python is (a*b)*c, sums of squares over the component axis are
//   sequential, numpy.maximum/minimum propagate NaN, masks follow the
//   reference's precedence.
// float — the bulk FP32 path.  Same formulas, rearranged for throughput:
//   one reciprocal per density instead of one division per use, approximate
//   division and square root (MUFU), NaN-propagating min/max in one
//   instruction, a single finiteness test per state.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "tfv_pair.cuh"
#include "tfv_soft64.cuh"

namespace tfv {

constexpr double kFloor = 1e-12;  // density / pressure floor
constexpr double kGuard = 1e-14;  // division guard (limiters, HLLC)

template <typename R>
struct Exact {
  static constexpr bool value = false;
};
template <>
struct Exact<double> {
  static constexpr bool value = true;
};

// numpy.maximum / numpy.minimum: NaN propagates, first operand wins ties.
// Double precision: integer comparisons (tfv_soft64.cuh), not the FP64 pipe.
__device__ __forceinline__ double np_max(double a, double b) { return soft_max(a, b); }
__device__ __forceinline__ double np_min(double a, double b) { return soft_min(a, b); }
__device__ __forceinline__ float np_max(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float np_min(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// numpy.maximum(a, numpy.maximum(b, c)) in one instruction: NaN if any
// operand is NaN (three-operand max, sm_100 and later).
__device__ __forceinline__ float np_max3(float a, float b, float c) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// a / b: IEEE division (double, on the integer pipe) or the approximate
// single-precision one.
__device__ __forceinline__ double dv(double a, double b) { return soft_div(a, b); }
__device__ __forceinline__ float dv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ float rcp(float b) { return __fdividef(1.0f, b); }
// a / b as the operator: IEEE (double), the unit's division flags (float).
__device__ __forceinline__ double qd(double a, double b) { return soft_div(a, b); }
__device__ __forceinline__ float qd(float a, float b) { return a / b; }
// a divisor used several times (double: its reciprocal estimate formed once)
template <typename R>
struct Divisor {
  R b;
  __device__ __forceinline__ explicit Divisor(R b_) : b(b_) {}
};
template <>
struct Divisor<double> {
  SoftDivisor d;
  __device__ __forceinline__ explicit Divisor(double b) : d(soft_divisor(b)) {}
};
__device__ __forceinline__ double qd(double a, const Divisor<double>& d) { return soft_div(a, d.d); }
__device__ __forceinline__ float qd(float a, const Divisor<float>& d) { return a / d.b; }
__device__ __forceinline__ double rt(double x) { return soft_sqrt(x); }
__device__ __forceinline__ float rt(float x) { return sqrtf(x); }
// x / 2 and 2 x, exact
__device__ __forceinline__ double hf(double x) { return soft_half(x); }
__device__ __forceinline__ float hf(float x) { return 0.5f * x; }
__device__ __forceinline__ double tw(double x) { return soft_twice(x); }
__device__ __forceinline__ float tw(float x) { return 2.0f * x; }
// comparisons (false for NaN)
__device__ __forceinline__ bool lt_(double a, double b) { return soft_lt(a, b); }
__device__ __forceinline__ bool lt_(float a, float b) { return a < b; }
__device__ __forceinline__ bool le_(double a, double b) { return soft_le(a, b); }
__device__ __forceinline__ bool le_(float a, float b) { return a <= b; }
__device__ __forceinline__ bool le0(double x) { return soft_le0(x); }
__device__ __forceinline__ bool le0(float x) { return x <= 0.0f; }
__device__ __forceinline__ bool ge0(double x) { return soft_ge0(x); }
__device__ __forceinline__ bool ge0(float x) { return x >= 0.0f; }
__device__ __forceinline__ bool gt0(double x) { return soft_gt0(x); }
__device__ __forceinline__ bool gt0(float x) { return x > 0.0f; }
__device__ __forceinline__ bool lt0(double x) { return soft_lt0(x); }
__device__ __forceinline__ bool lt0(float x) { return x < 0.0f; }
// x > c and |x| < c for a positive compile-time constant c
__device__ __forceinline__ bool gt_pos(double x, double c) { return soft_gt_pos(x, c); }
__device__ __forceinline__ bool gt_pos(float x, float c) { return x > c; }
__device__ __forceinline__ bool abs_lt(double x, double c) { return soft_abs_lt(x, c); }
__device__ __forceinline__ bool abs_lt(float x, float c) { return fabsf(x) < c; }
// np_max(x, c) for a positive compile-time constant c
__device__ __forceinline__ double max_pos(double x, double c) { return soft_max_pos(x, c); }
__device__ __forceinline__ float max_pos(float x, float c) { return np_max(x, c); }
template <typename R>
__device__ __forceinline__ R floored(R x) { return max_pos(x, R(kFloor)); }
// fmax(m, x) of a running maximum m >= 0
__device__ __forceinline__ double run_max(double m, double x) { return soft_fmax_run(m, x); }
__device__ __forceinline__ float run_max(float m, float x) { return fmaxf(m, x); }

// np.where(abs(x) < g, g, x), g a positive compile-time constant
template <typename R>
__device__ __forceinline__ R guarded(R x, R g) { return abs_lt(x, g) ? g : x; }

__device__ __forceinline__ bool finite_(double x) { return soft_isfinite(x); }
__device__ __forceinline__ bool finite_(float x) { return isfinite(x); }

// Constant gamma of an instance descriptor in the arithmetic type: single
// precision reads its float copy instead of converting the double per cell
// (a double-to-float conversion runs on the narrow FP64 pipe).
template <typename D>
__device__ __forceinline__ double desc_gamma(const D& d, double) { return d.gamma; }
template <typename D>
__device__ __forceinline__ float desc_gamma(const D& d, float) { return d.gamma_f; }

// --------------------------------------------------------------------------
// Limiters (LIM: 0 VanLeer, 1 Albada, 2 MINBEE, 3 Superbee, 4 Unos).
// 3D: python/cfdSolver/torchSolver3D.py:86-111.
// 2D: python/cfdSolver/torchSolver2D.py:124-168 (VanLeer/Albada zero for
//     r <= 0, Unos without the (1+2r)/3 bound).
// --------------------------------------------------------------------------
template <typename R, int DIM, int LIM>
__device__ __forceinline__ R limited_slope(R um, R uc, R up) {
  const R minus = uc - um;
  const R plus = up - uc;
  if constexpr (!Exact<R>::value && (LIM == 2 || LIM == 3)) {
    // single precision, MINBEE and Superbee: phi(r) * plus with r = minus /
    // plus, multiplied through by |plus| (no division): with s = sign(plus),
    // a = s * minus and b = |plus|, MINBEE is s * max(0, min(a, b)) and
    // Superbee s * max(0, max(min(2a, b), min(a, 2b))).  Equal to the
    // reference's form except where |plus| < 1e-14, whose guard changes the
    // result by less than 2e-14 (below single-precision resolution);
    // NaN still propagates through the NaN-propagating min / max.
    const R s = copysignf(1.0f, plus);
    const R a = minus * s;
    const R b = fabsf(plus);
    R t;
    if (LIM == 2)
      t = np_max(R(0), np_min(a, b));
    else
      t = np_max3(R(0), np_min(a + a, b), np_min(a, b + b));
    return t * s;
  }
  if constexpr (!Exact<R>::value && LIM == 0) {
    // single precision, VanLeer: with r = minus / plus > 0,
    // phi(r) * plus = 2 minus plus / (minus + plus); zero for r <= 0.  One
    // reciprocal instead of two; the guard of tiny |plus| makes a difference
    // below single-precision resolution; NaN inputs give NaN.
    const R mp = minus * plus;
    const R v = (mp + mp) * rcp(minus + plus);
    return mp > R(0) ? v : (mp == mp ? R(0) : mp);
  }
  // a divisor within the guard leaves |phi plus| below 1.2e-14 whatever stands in for
  // it; in single precision a large one, so that Albada's r^2 stays finite (a
  // pressure step of 5e5 Pa over 1e-14 does not)
  const R r = dv(minus, abs_lt(plus, R(kGuard)) ? R(Exact<R>::value ? kGuard : 1e18) : plus);
  R phi;
  if constexpr (Exact<R>::value) {
    phi = limiter_phi<DIM, LIM>(r);
  } else if (LIM == 1) {  // Albada
    const R pos = np_max(r, R(0));
    phi = dv(pos * pos + pos, pos * pos + R(1));
    if (DIM == 2 && !(r > R(0))) phi = R(0);
  } else {  // Unos (MINBEE, Superbee and VanLeer returned above)
    phi = np_min(np_min(R(2), R(2) * r), dv(R(2) + r, R(3)));
    if (DIM == 3) phi = np_min(phi, dv(R(1) + R(2) * r, R(3)));
    phi = np_max(R(0), phi);
  }
  return phi * plus;
}

// --------------------------------------------------------------------------
// Predictor fluxes.
// 3D _flux: python/cfdSolver/torchSolver3D.py:77-83 with uconsv_to_uprim_3d
//   (:37-44, no floors).  m = normal momentum row (1..3).
// 2D euler_flux_x / euler_flux_y: python/cfdSolver/torchSolver2D.py:326-352
//   (rho and p floored).
// --------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ void flux3(const R* u, R g, int m, R* f) {
  const R ssum = (u[1] * u[1] + u[2] * u[2]) + u[3] * u[3];
  R p, vel;
  if constexpr (Exact<R>::value) {
    const Divisor<R> rho(u[0]);
    p = (g - R(1)) * (u[4] - qd(hf(ssum), rho));
    vel = qd(u[m], rho);
  } else {
    const R irho = rcp(u[0]);
    p = (g - R(1)) * (u[4] - R(0.5) * ssum * irho);
    vel = u[m] * irho;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) f[c] = u[c] * vel;
  if constexpr (!Exact<R>::value) f[0] = u[m];  // rho * (m / rho) is the momentum itself
  f[m] = f[m] + p;
  f[4] = vel * (u[4] + p);
}

// flux3 of two states in packed arithmetic, single precision.
__device__ __forceinline__ void flux3_pair(const float* ua, const float* ub, float g, int m,
                                           float* fa, float* fb) {
  Pair u[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) u[c] = pk(ua[c], ub[c]);
  const Pair ssum = fma2(u[3], u[3], fma2(u[2], u[2], u[1] * u[1]));
  const Pair ir = pk(rcp(ua[0]), rcp(ub[0]));
  const Pair p = pk(g - 1.0f) * fma2(ssum * pk(-0.5f), ir, u[4]);
  const Pair vel = u[m] * ir;
  fa[0] = ua[m];
  fb[0] = ub[m];
#pragma unroll
  for (int c = 1; c < 4; ++c) {
    const Pair f = c == m ? fma2(u[c], vel, p) : u[c] * vel;
    unpk(f, fa[c], fb[c]);
  }
  unpk(vel * (u[4] + p), fa[4], fb[4]);
}

template <typename R>
__device__ __forceinline__ void flux2(const R* u, R g, int normal, R* f) {
  const R rho = floored(u[0]);
  R vx, vy;
  if constexpr (Exact<R>::value) {
    const Divisor<R> dr(rho);
    vx = qd(u[1], dr);
    vy = qd(u[2], dr);
  } else {
    const R irho = rcp(rho);
    vx = u[1] * irho;
    vy = u[2] * irho;
  }
  const R p = floored((g - R(1)) * (u[3] - hf(rho) * (vx * vx + vy * vy)));
  if (normal == 0) {
    f[0] = rho * vx;
    f[1] = rho * (vx * vx) + p;
    f[2] = (rho * vx) * vy;
    f[3] = vx * (u[3] + p);
  } else {
    f[0] = rho * vy;
    f[1] = (rho * vx) * vy;
    f[2] = rho * (vy * vy) + p;
    f[3] = vy * (u[3] + p);
  }
}

// flux2 of two states in packed arithmetic, single precision.
__device__ __forceinline__ void flux2_pair(const float* ua, const float* ub, float g, int normal,
                                           float* fa, float* fb) {
  const float ra = floored(ua[0]), rb = floored(ub[0]);
  const Pair r = pk(ra, rb), ir = pk(rcp(ra), rcp(rb)), e = pk(ua[3], ub[3]);
  const Pair vx = pk(ua[1], ub[1]) * ir, vy = pk(ua[2], ub[2]) * ir;
  const Pair pe = pk(g - 1.0f) * fma2(r * pk(-0.5f), fma2(vy, vy, vx * vx), e);
  const Pair p = pk(floored(lo_(pe)), floored(hi_(pe)));
  const Pair vn = normal == 0 ? vx : vy;
  const Pair mx = r * vx;
  if (normal == 0) {
    unpk(mx, fa[0], fb[0]);
    unpk(fma2(mx, vx, p), fa[1], fb[1]);
    unpk(mx * vy, fa[2], fb[2]);
  } else {
    const Pair my = r * vy;
    unpk(my, fa[0], fb[0]);
    unpk(mx * vy, fa[1], fb[1]);
    unpk(fma2(my, vy, p), fa[2], fb[2]);
  }
  unpk(vn * (e + p), fa[3], fb[3]);
}

// Physical-state test of one cell (python/cfdSolver/torchSolver.py:1038-1046).
template <typename R, int NV>
__device__ __forceinline__ bool physical_cell(const R* u) {
  R s = u[1] * u[1];
#pragma unroll
  for (int c = 2; c < NV - 1; ++c) s = s + u[c] * u[c];
  if constexpr (Exact<R>::value) {
    bool ok = true;
#pragma unroll
    for (int c = 0; c < NV; ++c) ok = ok & finite_(u[c]);
    return ok & gt_pos(u[0], R(kFloor)) & gt_pos(u[NV - 1] - qd(hf(s), u[0]), R(kFloor));
  } else {
    // one finiteness test: any NaN or infinity makes the sum non-finite
    R all = u[0];
#pragma unroll
    for (int c = 1; c < NV; ++c) all = all + u[c];
    // E - |m|^2 / (2 rho) > floor, multiplied through by rho > floor
    return finite_(all) && (u[0] > R(kFloor)) &&
           (u[NV - 1] * u[0] - R(0.5) * s > R(kFloor) * u[0]);
  }
}

// --------------------------------------------------------------------------
// HLLC in the normal basis: rows rho, m_n, m_t[NT], E
// (python/cfdSolver/torchFlux.py:125-248).  Only the star state of the side
// that can be selected is formed; values are identical to evaluating both.
// Where no wave-speed mask holds (NaN speeds) the result is NaN.
// --------------------------------------------------------------------------
// Double precision: only the flux and the star state of the side that the
// masks select are formed (values identical to evaluating both).
template <int NT>
__device__ __forceinline__ void hllc_f64(const double* ul, const double* ur, double gl, double gr,
                                         double* out) {
  using R = double;
  constexpr int NV = NT + 3;
  constexpr int E = NV - 1;
  const R g = hf(gl + gr);
  const R rl = floored(ul[0]);
  const R rr = floored(ur[0]);
  const Divisor<R> dl(rl), dr(rr);
  const R unl = qd(ul[1], dl);
  const R unr = qd(ur[1], dr);
  R utl[NT], utr[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    utl[t] = qd(ul[2 + t], dl);
    utr[t] = qd(ur[2 + t], dr);
  }
  R stl = utl[0] * utl[0], str = utr[0] * utr[0];
#pragma unroll
  for (int t = 1; t < NT; ++t) {
    stl = stl + utl[t] * utl[t];
    str = str + utr[t] * utr[t];
  }
  const R kel = hf(rl) * (unl * unl + stl);
  const R ker = hf(rr) * (unr * unr + str);
  const R pl = floored((gl - R(1)) * (ul[E] - kel));
  const R pr = floored((gr - R(1)) * (ur[E] - ker));
  const R al = rt(qd(gl * pl, dl));
  const R ar = rt(qd(gr * pr, dr));

  const R sql = rt(rl);
  const R sqr = rt(rr);
  const R inv = qd(R(1), sql + sqr);
  const R uroe = (sql * unl + sqr * unr) * inv;
  R vsum;
  {
    const R v0 = (sql * utl[0] + sqr * utr[0]) * inv;
    vsum = v0 * v0;
#pragma unroll
    for (int t = 1; t < NT; ++t) {
      const R vt = (sql * utl[t] + sqr * utr[t]) * inv;
      vsum = vsum + vt * vt;
    }
  }
  const R epl = ul[E] + pl, epr = ur[E] + pr;
  const R hl = qd(epl, dl);
  const R hr = qd(epr, dr);
  const R hroe = (sql * hl + sqr * hr) * inv;
  const R keroe = hf(uroe * uroe + vsum);
  const R aroe = rt(floored((g - R(1)) * (hroe - keroe)));

  const R sL = np_min(unl - al, uroe - aroe);
  const R sR = np_max(unr + ar, uroe + aroe);
  const R den = guarded(rl * (sL - unl) - rr * (sR - unr), R(kGuard));
  const R ss = dv(((pr - pl) + (rl * unl) * (sL - unl)) - (rr * unr) * (sR - unr), den);

  const bool mr = le0(sR);
  const bool ssn = le0(ss);
  const bool mstar = (ssn && ge0(sR)) || (le0(sL) && ge0(ss));
  const bool ml = ge0(sL);
  // the side whose flux the selected region reads (right supersonic, then the
  // star region of the side ss picks, then left supersonic)
  const bool right = mr || (mstar && ssn);
  const R rho = right ? rr : rl;
  const R un = right ? unr : unl;
  const R p = right ? pr : pl;
  const R s = right ? sR : sL;
  const R uE = right ? ur[E] : ul[E];
  R f[NV];
  f[0] = rho * un;
  f[1] = rho * (un * un) + p;
#pragma unroll
  for (int t = 0; t < NT; ++t) f[2 + t] = (rho * un) * (right ? utr[t] : utl[t]);
  f[E] = un * (right ? epr : epl);
  const R gap = s - ss;
  if (!mr && mstar && !abs_lt(gap, R(kFloor))) {  // star state of that side
    const R dss = guarded(gap, R(kGuard));
    const R rho_s = floored(rho * dv(s - un, dss));
    const R dun = guarded(s - un, R(kGuard));
    R star[NV];
    star[0] = rho_s;
    star[1] = rho_s * ss;
#pragma unroll
    for (int t = 0; t < NT; ++t) star[2 + t] = rho_s * (right ? utr[t] : utl[t]);
    star[E] = rho_s * (qd(uE, right ? dr : dl) + (ss - un) * (ss + qd(p, rho * dun)));
#pragma unroll
    for (int c = 0; c < NV; ++c) f[c] = f[c] + s * (star[c] - (right ? ur[c] : ul[c]));
  }
#pragma unroll
  for (int c = 0; c < NV; ++c) out[c] = (mr || mstar || ml) ? f[c] : R(NAN);
}

// Single precision: both physical fluxes (measured faster in 2D).
template <int NT>
__device__ __forceinline__ void hllc_f32(const float* ul, const float* ur, float gl, float gr,
                                         float* out) {
  using R = float;
  constexpr int NV = NT + 3;
  constexpr int E = NV - 1;
  // the two sides are the halves of packed pairs
  const R g = R(0.5) * (gl + gr);
  const R rl = np_max(ul[0], R(kFloor));
  const R rr = np_max(ur[0], R(kFloor));
  const R irl = rcp(rl), irr = rcp(rr);
  const Pair r = pk(rl, rr), ir = pk(irl, irr), e = pk(ul[E], ur[E]);
  const Pair un2 = pk(ul[1], ur[1]) * ir;
  Pair ut[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) ut[t] = pk(ul[2 + t], ur[2 + t]) * ir;
  Pair q = ut[0] * ut[0];
#pragma unroll
  for (int t = 1; t < NT; ++t) q = fma2(ut[t], ut[t], q);
  q = fma2(un2, un2, q);
  const Pair ei = fma2(r * pk(-0.5f), q, e);  // internal energy density
  const R pl = np_max((gl - R(1)) * lo_(ei), R(kFloor));
  const R pr = np_max((gr - R(1)) * hi_(ei), R(kFloor));
  const Pair p2 = pk(pl, pr);
  const Pair a2 = (pk(gl, gr) * p2) * ir;
  const R al = sqrtf(lo_(a2)), ar = sqrtf(hi_(a2));
  const Pair ep = e + p2;

  const Pair mn = r * un2;
  R fl[NV], fr[NV];
  unpk(mn, fl[0], fr[0]);
  unpk(fma2(mn, un2, p2), fl[1], fr[1]);
#pragma unroll
  for (int t = 0; t < NT; ++t) unpk(mn * ut[t], fl[2 + t], fr[2 + t]);
  unpk(un2 * ep, fl[E], fr[E]);

  const R sql = sqrtf(rl), sqr = sqrtf(rr);
  const R inv = rcp(sql + sqr);
  const R wl = sql * inv, wr = sqr * inv;  // Roe weights
  const R unl = lo_(un2), unr = hi_(un2);
  R utl[NT], utr[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) unpk(ut[t], utl[t], utr[t]);
  const R uroe = wl * unl + wr * unr;
  R vsum = uroe * uroe;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const R vt = wl * utl[t] + wr * utr[t];
    vsum = vsum + vt * vt;
  }
  const Pair h = ep * ir;
  const R hroe = wl * lo_(h) + wr * hi_(h);
  const R aroe = sqrtf(np_max((g - R(1)) * (hroe - R(0.5) * vsum), R(kFloor)));

  const R sL = np_min(unl - al, uroe - aroe);
  const R sR = np_max(unr + ar, uroe + aroe);
  const Pair m = r * (pk(sL, sR) - un2);
  const R den = guarded(lo_(m) - hi_(m), R(kGuard));
  const R ss = dv(((pr - pl) + unl * lo_(m)) - unr * hi_(m), den);

  // star state of the side whose star region can be selected
  const bool right = (ss <= R(0));
  const R rho = right ? rr : rl;
  const R un = right ? unr : unl;
  const R p = right ? pr : pl;
  const R s = right ? sR : sL;
  const R uE = right ? ur[E] : ul[E];
  const R dss = guarded(s - ss, R(kGuard));
  const R rho_s = np_max(rho * dv(s - un, dss), R(kFloor));
  const R dun = guarded(s - un, R(kGuard));
  R star[NV];
  star[0] = rho_s;
  star[1] = rho_s * ss;
#pragma unroll
  for (int t = 0; t < NT; ++t) star[2 + t] = rho_s * (right ? utr[t] : utl[t]);
  star[E] = rho_s * (uE * (right ? irr : irl) + (ss - un) * (ss + dv(p, rho * dun)));
  const bool close = fabs(s - ss) < R(kFloor);

  const bool mr = (R(0) >= sR);
  const bool msr = (ss <= R(0)) && (R(0) <= sR);
  const bool msl = (sL <= R(0)) && (R(0) <= ss);
  const bool ml = (R(0) <= sL);
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    const R uc = right ? ur[c] : ul[c];
    const R fc = right ? fr[c] : fl[c];
    const R fstar = close ? fc : fc + s * (star[c] - uc);
    R v = R(NAN);
    if (ml) v = fl[c];
    if (msl || msr) v = fstar;
    if (mr) v = fr[c];
    out[c] = v;
  }
}

template <typename R, int NT>
__device__ __forceinline__ void hllc(const R* ul, const R* ur, R gl, R gr, R* out) {
  if constexpr (Exact<R>::value)
    hllc_f64<NT>(ul, ur, gl, gr, out);
  else
    hllc_f32<NT>(ul, ur, gl, gr, out);
}

// Rotation into the normal basis (python/cfdSolver/torchFlux.py:36-39):
// order = [0, normal] + other momenta ascending + [E].
template <int NV>
__device__ __forceinline__ void normal_order(int normal, int* order) {
  order[0] = 0;
  order[1] = normal;
  int k = 2;
#pragma unroll
  for (int m = 1; m < NV - 1; ++m)
    if (m != normal) order[k++] = m;
  order[NV - 1] = NV - 1;
}

// Single-precision HLLC of the fused step (same states, speeds and masks as
// hllc above).  Only one physical flux is formed: the region that the masks
// select (left, right, or the star state of the side `ss <= 0` picks, in the
// reference's precedence: right supersonic, then star, then left
// supersonic) reads one side's flux, so the other side's flux is never
// needed.  It also tests both input face states for the 3D predictor gate
// (density and internal energy density above the floor; NaN fails) and ORs
// the result into `gate`: every predicted face state the step consumes
// passes through here once.  NaN where no mask holds, as in hllc.
template <int NT>
__device__ __forceinline__ void hllc_gated(const float* ul, const float* ur, float gl, float gr,
                                           float* out, bool& gate) {
  constexpr int NV = NT + 3;
  constexpr int E = NV - 1;
  const float fl = float(kFloor);
  const float g = 0.5f * (gl + gr);
  // the two sides are the halves of packed pairs up to the wave speeds.  The
  // density floors of the reference change nothing here: a face state
  // whose density is not above the floor fails the gate test below and the
  // step is redone to first order
  const Pair r = pk(ul[0], ur[0]), e = pk(ul[E], ur[E]);
  const float irl = rcp(ul[0]), irr = rcp(ur[0]);
  const Pair ir = pk(irl, irr);
  const Pair un = pk(ul[1], ur[1]) * ir;
  Pair ut[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) ut[t] = pk(ul[2 + t], ur[2 + t]) * ir;
  Pair q = ut[0] * ut[0];
#pragma unroll
  for (int t = 1; t < NT; ++t) q = fma2(ut[t], ut[t], q);
  q = fma2(un, un, q);
  const Pair ei = fma2(r * pk(-0.5f), q, e);  // internal energy density
  float eil, eir;
  unpk(ei, eil, eir);
  if (!(ul[0] > fl && eil > fl && ur[0] > fl && eir > fl)) gate = true;
  const float pl = np_max((gl - 1.0f) * eil, fl);
  const float pr = np_max((gr - 1.0f) * eir, fl);
  const Pair p2 = pk(pl, pr);
  const Pair a2 = (pk(gl, gr) * p2) * ir;
  const float al = sqrtf(lo_(a2)), ar = sqrtf(hi_(a2));
  const float sql = sqrtf(ul[0]), sqr = sqrtf(ur[0]);
  const float inv = rcp(sql + sqr);
  const float wl = sql * inv, wr = sqr * inv;  // Roe weights
  const float unl = lo_(un), unr = hi_(un);
  const float uroe = wl * unl + wr * unr;
  float vsum = uroe * uroe;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const float vt = wl * lo_(ut[t]) + wr * hi_(ut[t]);
    vsum = vsum + vt * vt;
  }
  const Pair h = (e + p2) * ir;
  const float hroe = wl * lo_(h) + wr * hi_(h);
  const float aroe = sqrtf(np_max((g - 1.0f) * (hroe - 0.5f * vsum), fl));
  const float sL = np_min(unl - al, uroe - aroe);
  const float sR = np_max(unr + ar, uroe + aroe);
  const Pair gap = pk(sL, sR) - un;
  const Pair m = r * gap;
  const float ml_ = lo_(m), mr_ = hi_(m);
  const float den = guarded(ml_ - mr_, float(kGuard));
  const float ss = dv(((pr - pl) + unl * ml_) - unr * mr_, den);

  const bool mr = (0.0f >= sR);
  const bool mstar = ((ss <= 0.0f) && (0.0f <= sR)) || ((sL <= 0.0f) && (0.0f <= ss));
  const bool ml = (0.0f <= sL);
  // side whose flux the selected region reads
  const bool right = mr || (mstar && ss <= 0.0f);
  const float irho = right ? irr : irl;
  const float v = right ? unr : unl;
  const float p = right ? pr : pl;
  float u[NV], f[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) u[c] = right ? ur[c] : ul[c];
  // rho * (m / rho), not the momentum row itself: over 200 steps of the 256^3
  // explosion the L1 error of rho is 1.62e-8 with it and 1.79e-8 without
  const float mn = u[0] * v;
  f[0] = mn;
  f[1] = mn * v + p;
#pragma unroll
  for (int t = 0; t < NT; ++t) f[2 + t] = mn * (right ? hi_(ut[t]) : lo_(ut[t]));
  f[E] = v * (u[E] + p);
  const float s = right ? sR : sL;
  if (!mr && mstar && !(fabsf(s - ss) < fl)) {
    const float rho_s = np_max(u[0] * dv(s - v, guarded(s - ss, float(kGuard))), fl);
    const float dun = guarded(s - v, float(kGuard));
    float star[NV];
    star[0] = rho_s;
    star[1] = rho_s * ss;
#pragma unroll
    for (int t = 0; t < NT; ++t) star[2 + t] = rho_s * (right ? hi_(ut[t]) : lo_(ut[t]));
    star[E] = rho_s * (u[E] * irho + (ss - v) * (ss + dv(p, u[0] * dun)));
#pragma unroll
    for (int c = 0; c < NV; ++c) f[c] = f[c] + s * (star[c] - u[c]);
  }
  // No NaN select for "no region": with face states that pass the gate test
  // above, sL, sR and ss are finite and one of the three regions always
  // holds; states that fail it flag the tile, and the flagged step is redone
  // to first order, so this flux is never committed.
#pragma unroll
  for (int c = 0; c < NV; ++c) out[c] = f[c];
}

template <int NV>
__device__ __forceinline__ void hllc_cartesian_gated(const float* L, const float* Rt, float gl,
                                                     float gr, int d, float* F, bool& gate) {
  int order[NV];
  normal_order<NV>(d + 1, order);
  float ul[NV], ur[NV], f[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    ul[c] = L[order[c]];
    ur[c] = Rt[order[c]];
  }
  hllc_gated<NV - 3>(ul, ur, gl, gr, f, gate);
#pragma unroll
  for (int c = 0; c < NV; ++c) F[order[c]] = f[c];
}

// HLLC across a face along direction d (0=x,1=y,2=z) with Cartesian inputs
// and output (python/cfdSolver/torchFlux.py:6-77 without the batching).
template <typename R, int NV>
__device__ __forceinline__ void hllc_cartesian(const R* L, const R* Rt, R gl, R gr, int d,
                                               R* F) {
  int order[NV];
  normal_order<NV>(d + 1, order);
  R ul[NV], ur[NV], f[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    ul[c] = L[order[c]];
    ur[c] = Rt[order[c]];
  }
  hllc<R, NV - 3>(ul, ur, gl, gr, f);
#pragma unroll
  for (int c = 0; c < NV; ++c) F[order[c]] = f[c];
}

}  // namespace tfv
