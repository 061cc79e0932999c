// g5_fast64.cuh — the FP64 form's per-cell arithmetic for the stiffened-gas
// mixture with as few FP64-pipe instructions as its results allow.
//
// The reference arithmetic (prim_fp64, hllc_fp64, slope_scalar<double>,
// update_fp64 in g5_common.cuh and g5_step2d.cuh) is bound by the FP64 pipe:
// 1.66 instructions per clock per SM on GB300, two orders of magnitude below
// the integer and FP32 pipes.  The functions here return the same doubles
// (compared bit for bit with the CPU oracle; only the sign of a zero may
// differ) from fewer of them:
//   * divisions and square roots on the integer pipes (g5_exact64.h), the
//     quotients of one divisor sharing its reciprocal;
//   * about half of the products on the integer pipes (mul64: 0.56 clocks per
//     product and SM against 0.60 for the FP64 pipe, which runs beside them;
//     the split was found by moving groups of products: all of them on the
//     integer pipes is 8 % slower, the kinetic energies', the HLLC averages' or
//     the dt/dx scaling back on the FP64 pipe 2 to 3 % each);
//   * comparisons, minima, maxima, clamps and sign tests on bit patterns;
//   * factors of 1/2 folded into one fused multiply-add (x +- y/2 rounds once,
//     as a separate, exact y/2 would) or carried to the next such addition;
//   * sqrt(fl(c^2)) = c (Boldo 2015: exact in radix 2 without over- or
//     underflow), which removes two square roots per face;
//   * minmod slopes without the central difference: when both one-sided
//     differences agree in sign, |q+ - q-|/2 is never below the smaller one
//     (rounding is monotonic), so it never limits;
//   * terms that vanish for the case at hand (pinf = 0).
// Every shortcut assumes values that are zero or within 2^-900 .. 2^700
// (g5_exact64.h): states read from memory are tested, results set `bad` when
// they leave the range, and the caller then evaluates with the reference
// functions.
#pragma once

#include "g5_common.cuh"
#include "g5_exact64.h"
#include "g5_mg64.cuh"

namespace g5
{

__device__ __forceinline__ long long
bits64(double x)
{
  return __double_as_longlong(x);
}

// a bit pattern that orders doubles as signed integers (-0 just below +0)
__device__ __forceinline__ long long
order64(double x)
{
  const long long b = bits64(x);
  return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL);
}

// -x without the FP64 pipe (a selected -x is a subtraction from -0 there)
__device__ __forceinline__ double
neg64(double x)
{
  return x64_make(x64_hi(x) ^ 0x80000000u, x64_lo(x));
}

// x + y where `on`, else x: under a predicate, so that the FP64 pipe has no
// work where it is off (an ordinary conditional sum is computed and selected)
__device__ __forceinline__ double
add_if64(bool on, double x, double y)
{
  double r = x;
  asm volatile("{.reg .pred p; setp.ne.u32 p, %2, 0; @p add.rn.f64 %0, %0, %1;}" : "+d"(r) : "d"(y), "r"((unsigned)on));
  return r;
}

// a / b in hardware, off the main path
static __device__ __noinline__ double
div_cold64(double a, double b)
{
  return a / b;
}

// max(x, c) for c > 0, x no NaN
__device__ __forceinline__ double
max_pos64(double x, double c)
{
  return bits64(x) > bits64(c) ? x : c;
}

// x where it is positive, else +0
__device__ __forceinline__ double
clip0_64(double x)
{
  return bits64(x) > 0 ? x : 0.0;
}

// a b on the FP64 pipe, with the range test of mul64
__device__ __forceinline__ double
mulh64(double a, double b, bool & bad)
{
  const double r = a * b;
  bad = bad || x64_raw_bad(r);
  return r;
}

// PI = a0 gpx0 + a1 gpx1 of the stiffened-gas mixture, the terms of a zero
// constant left out
__device__ __forceinline__ double
mix_PI64(const PhysParams & P, double a0, double a1, bool & bad)
{
  if (P.pi64 == 3)
    return mul64(a0, P.gpx[0], bad) + mul64(a1, P.gpx[1], bad);
  return P.pi64 == 0 ? 0.0 : (P.pi64 == 1 ? mul64(a0, P.gpx[0], bad) : mul64(a1, P.gpx[1], bad));
}

__device__ __forceinline__ double
mix_S64(const PhysParams & P, double a0, double a1, bool & bad)
{
  return mul64(a0, P.xi[0], bad) + mul64(a1, P.xi[1], bad);
}

// the mixture rules (MG: the general ones of g5_mg64.cuh)
template <bool MG>
__device__ __forceinline__ Mix64
mixture64(const PhysParams & P, double a0, double a1, double ar0, double ar1, bool & bad)
{
  Mix64 m;
  if constexpr (MG)
  {
    const MixBad64 r = mg_mixture_fast64(&P, a0, a1, ar0, ar1);
    m = r.m;
    bad = bad || r.bad;
  }
  else
  {
    m.S = mix_S64(P, a0, a1, bad);
    m.PI = m.C0 = mix_PI64(P, a0, a1, bad);
    m.C1 = m.S + 1.0;
  }
  return m;
}

// whether the mixture has a PI and a C0
template <bool MG>
__device__ __forceinline__ bool
mixture_stiff64(const PhysParams & P)
{
  return MG || P.pi64 != 0;
}

// c = sqrt((p C1 + C0) / (rho S)), clipped at 0
__device__ __forceinline__ double
sound64(double rho, double p, const Mix64 & m, bool stiff, bool & bad)
{
  const double n = add_if64(stiff, mul64(p, m.C1, bad), m.C0);
  return sqrt64(clip0_64(div64(n, mul64(rho, m.S, bad), bad)), bad);
}

// clamps of computePrimitives: a partial density below 1e-12, and the volume
// fraction to [0, 1] with its ends widened by 1e-12
__device__ __forceinline__ double
clamp_r64(double r)
{
  return bits64(r) < bits64(1e-12) ? 0.0 : r;
}

__device__ __forceinline__ double
clamp_a64(double a)
{
  double r = bits64(a) < bits64(1e-12) ? 0.0 : a;
  return bits64(r) > bits64(1.0 - 1e-12) ? 1.0 : r;
}

// prim_fp64 (stiffened gases); the sound speed only when asked for.  RAW: the
// state comes from memory
template <int DIM, bool SOUND, bool RAW, bool MG>
__device__ __forceinline__ double
prim_fast64(const double * u, double * q, const PhysParams & P, bool & bad)
{
  using H = V<DIM>;
  const bool    stiff = mixture_stiff64<MG>(P);
  const double  d = max_pos64(u[H::ID], P.smallr);
  const Recip64 rd = recip64(d, bad);
  const double  ux = quot64(u[H::IU], rd, bad), uy = quot64(u[H::IV], rd, bad);
  double        k2 = mul64(ux, ux, bad) + mul64(uy, uy, bad), uz = 0.0;
  if constexpr (DIM == 3)
  {
    uz = quot64(u[H::IW], rd, bad);
    k2 = k2 + mul64(uz, uz, bad);
  }
  const double eint = __fma_rn(-0.5, k2, quot64(u[H::IE], rd, bad));
  const double a0u = u[H::IA0], a1u = 1.0 - a0u;
  Mix64        m = mixture64<MG>(P, a0u, a1u, u[H::IAD0], u[H::IAD1], bad);
  const double p = div64(add_if64(stiff, mul64(d, eint, bad), neg64(m.PI)), m.S, bad);
  const double a0 = clamp_a64(a0u);
  if constexpr (RAW)
  {
    bad = bad || x64_raw_bad(d) || x64_raw_bad(u[H::IE]) || x64_raw_bad(u[H::IU]) || x64_raw_bad(u[H::IV]) || x64_raw_bad(a0u) ||
          x64_raw_bad(u[H::IAD0]) || x64_raw_bad(u[H::IAD1]);
    if constexpr (DIM == 3)
      bad = bad || x64_raw_bad(u[H::IW]);
  }
  q[H::QR0] = clamp_r64(u[H::IAD0]);
  q[H::QR1] = clamp_r64(u[H::IAD1]);
  q[H::QP] = p;
  q[H::QU] = ux;
  q[H::QV] = uy;
  if constexpr (DIM == 3)
    q[H::QW] = uz;
  q[H::QA] = a0;
  if constexpr (SOUND)
  {
    // (the mixture of the clamped state)
    if (bits64(a0) != bits64(a0u) || (MG && (bits64(q[H::QR0]) != bits64(u[H::IAD0]) || bits64(q[H::QR1]) != bits64(u[H::IAD1]))))
      m = mixture64<MG>(P, a0, 1.0 - a0, q[H::QR0], q[H::QR1], bad);
    return sound64(d, p, m, stiff, bad);
  }
  return 0.0;
}

// slope_scalar<double> for slope_type 1 (minmod) and 2, from the one-sided
// differences l and r.  Their product, whose sign decides, is not formed: when it could
// underflow (the reference takes that as no slope) the cell is `bad`.
__device__ __forceinline__ double
limit_fast64(double l, double r, double qPlus, double qMinus, int st, bool & bad)
{
  const uint32_t hl = x64_hi(l), hr = x64_hi(r);
  const uint32_t el = hl & 0x7FF00000u, er = hr & 0x7FF00000u;
  const bool     same = (int)(hl ^ hr) >= 0 && el != 0u && er != 0u;
  bad = bad || (same && el + er < 0x3CC00000u); // |l r| may be below 2^-1074
  const unsigned long long al = (unsigned long long)bits64(l) << 1, ar = (unsigned long long)bits64(r) << 1;
  const bool               left = al < ar;
  double                   m = left ? l : r;
  if (st == 2)
  {
    // 2 min(|l|, |r|) against |q+ - q-| / 2
    const double c = qPlus - qMinus;
    m = m + m;
    const double h = 0.5 * c;
    m = ((unsigned long long)bits64(m) << 1) < ((unsigned long long)bits64(h) << 1) ? m : x64_make((x64_hi(h) & 0x7FFFFFFFu) | (x64_hi(m) & 0x80000000u), x64_lo(h));
  }
  // no slope: a zero with the sign of the central difference
  return same ? m : x64_make(order64(qPlus) >= order64(qMinus) ? 0u : 0x80000000u, 0u);
}

__device__ __forceinline__ double
slope_fast64(double q, double qPlus, double qMinus, int st, bool & bad)
{
  return limit_fast64(q - qMinus, qPlus - q, qPlus, qMinus, st, bad);
}

// HLLC (hllc_fp64) of two reconstructed states, scaled by dt/dx; S the
// mixture's of the side (stiffened gases; MG evaluates the mixture here).  f: FR0 FR1 FA0 FA1 FE FU FV (FW) FUS.
static __device__ __noinline__ double
floor_p64(double p, double r, double smallp)
{
  return fmax(p, r * smallp);
}

struct Side64
{
  double r, u, p, e, c; // density, normal velocity, pressure, total energy, sound speed (at least smallc)
};

template <int DIM, bool MG>
__device__ __forceinline__ Side64
hllc_side64(const double * q, double S, const PhysParams & P, bool & bad)
{
  using H = V<DIM>;
  const bool stiff = mixture_stiff64<MG>(P);
  Side64 s;
  s.r = max_pos64(q[H::QR0] + q[H::QR1], P.smallr);
  double p = q[H::QP];
  // max(p, r smallp): the product only where p is not far above it
  if ((int)x64_hi(p) <= (int)((x64_hi(s.r) & 0x7FF00000u) + (x64_hi(P.smallp) & 0x7FF00000u) - 0x3FD00000u))
    p = floor_p64(p, s.r, P.smallp);
  s.u = q[H::QU];
  Mix64 m;
  if constexpr (MG)
    m = mixture64<true>(P, q[H::QA], 1.0 - q[H::QA], q[H::QR0], q[H::QR1], bad);
  else
  {
    m.S = S;
    m.PI = m.C0 = stiff ? mix_PI64(P, q[H::QA], 1.0 - q[H::QA], bad) : 0.0;
    m.C1 = S + 1.0;
  }
  const double n = add_if64(stiff, mulh64(p, m.S, bad), m.PI);
  const double re = mulh64(s.r, div64(n, s.r, bad), bad); // rho e
  s.p = div64(add_if64(stiff, re, neg64(m.PI)), m.S, bad);
  double k = mul64(mul64(s.r, s.u, bad), s.u, bad) + mul64(mul64(s.r, q[H::QV], bad), q[H::QV], bad);
  if constexpr (DIM == 3)
    k = k + mul64(mul64(s.r, q[H::QW], bad), q[H::QW], bad);
  s.e = __fma_rn(0.5, k, re);
  const double c = sound64(s.r, s.p, m, stiff, bad);
  s.c = max_pos64(c, P.smallc);
  return s;
}

template <int DIM>
__device__ __forceinline__ void
hllc_fast64(const double * ql, const double * qr, const Side64 & L, const Side64 & R, double dtdx, double * f, bool & bad)
{
  using H = V<DIM>;
  const double cm = max_pos64(L.c, R.c);
  const bool   lo = order64(L.u) < order64(R.u);
  const double SL = (lo ? L.u : R.u) - cm;
  const double SR = (lo ? R.u : L.u) + cm;
  const double dl = L.u - SL, dr = SR - R.u;
  const double rcl = mul64(L.r, dl, bad), rcr = mul64(R.r, dr, bad);
  const Recip64 rs = recip64(rcr + rcl, bad);
  const double us = quot64((mul64(rcr, R.u, bad) + mul64(rcl, L.u, bad)) + (L.p - R.p), rs, bad);
  const double ps = quot64((mul64(rcr, L.p, bad) + mul64(rcl, R.p, bad)) + mul64(mul64(rcl, rcr, bad), L.u - R.u, bad), rs, bad);

  const bool left = bits64(SL) > 0 || bits64(us) > 0;
  double     r0 = left ? ql[H::QR0] : qr[H::QR0], r1 = left ? ql[H::QR1] : qr[H::QR1];
  double     ro = left ? L.r : R.r, uo = left ? L.u : R.u, po = left ? L.p : R.p, eo = left ? L.e : R.e;
  // between the outer waves: the star state of the upwind side
  if (!(bits64(SL) > 0) && (bits64(us) > 0 || bits64(SR) > 0))
  {
    const double  ds = left ? neg64(dl) : dr; // S - u
    const Recip64 rd = recip64((left ? SL : SR) - us, bad);
    const double  fac = quot64(ds, rd, bad);
    r0 = mulh64(r0, fac, bad);
    r1 = mulh64(r1, fac, bad);
    ro = mulh64(ro, fac, bad);
    eo = quot64((mulh64(ds, eo, bad) - mulh64(po, uo, bad)) + mulh64(ps, us, bad), rd, bad);
    uo = us;
    po = ps;
  }
  const double fid = mulh64(r0 + r1, uo, bad);
  const bool   up = bits64(fid) > 0;
  f[H::FR0] = mulh64(mulh64(r0, uo, bad), dtdx, bad);
  f[H::FR1] = mul64(mulh64(r1, uo, bad), dtdx, bad);
  f[H::FU] = mul64(mulh64(mul64(ro, uo, bad), uo, bad) + po, dtdx, bad);
  f[H::FE] = mul64(mulh64(eo + po, uo, bad), dtdx, bad);
  f[H::FV] = mul64(mulh64(fid, up ? ql[H::QV] : qr[H::QV], bad), dtdx, bad);
  if constexpr (DIM == 3)
    f[H::FW] = mul64(mulh64(fid, up ? ql[H::QW] : qr[H::QW], bad), dtdx, bad);
  const double phi0 = up ? ql[H::QA] : qr[H::QA];
  f[H::FA0] = mul64(mulh64(uo, phi0, bad), dtdx, bad);
  f[H::FA1] = mulh64(mulh64(uo, 1.0 - phi0, bad), dtdx, bad);
  f[H::FUS] = mul64(uo, dtdx, bad);
}

// source_factors_fp64 (MG: left to the reference arithmetic)
template <int DIM, bool MG>
__device__ __forceinline__ void
source_factors_fast64(const double * u, const PhysParams & P, double & st0, double & st1, bool & bad)
{
  using H = V<DIM>;
  st0 = st1 = 1.0;
  if (P.source_term != 1)
    return;
  if constexpr (MG)
  {
    bad = true;
    return;
  }
  const double  d = max_pos64(u[H::IAD0] + u[H::IAD1], P.smallr);
  const Recip64 rdd = recip64(max_pos64(u[H::ID], P.smallr), bad);
  const double  ux = quot64(u[H::IU], rdd, bad), uy = quot64(u[H::IV], rdd, bad);
  double        k2 = mul64(ux, ux, bad) + mul64(uy, uy, bad);
  if constexpr (DIM == 3)
  {
    const double uz = quot64(u[H::IW], rdd, bad);
    k2 = k2 + mul64(uz, uz, bad);
  }
  const double  eint = __fma_rn(-0.5, k2, div64(u[H::IE], d, bad));
  const double  a0 = u[H::IA0], a1 = 1.0 - a0;
  const double  p = div64(mul64(d, eint, bad) - mix_PI64(P, a0, a1, bad), mix_S64(P, a0, a1, bad), bad);
  const Recip64 r0 = recip64(mul64(P.gamma[0], p + P.pinf[0], bad), bad), r1 = recip64(mul64(P.gamma[1], p + P.pinf[1], bad), bad);
  const double  kbar = div64(1.0, quot64(a0, r0, bad) + quot64(u[H::IA1], r1, bad), bad);
  st0 = 1.0 - quot64(kbar, r0, bad);
  st1 = 1.0 - quot64(kbar, r1, bad);
}

// the volume-fraction increment ((F_left - s u*_left) - F_right) + s u*_right, s = st a
__device__ __forceinline__ double
alpha_inc64(double fl, double fr, double usl, double usr, double st, double a, bool mp, bool & bad)
{
  if (mp)
  {
    usl = mul64(st, usl, bad);
    usr = mul64(st, usr, bad);
  }
  return ((fl - mul64(usl, a, bad)) - fr) + mul64(usr, a, bad);
}

// end of the update: renormalised volume fractions and ID, then the new
// state's CFL rate (ComputeDtFiveEqFunctor) when asked for
template <int DIM, bool MG>
__device__ __forceinline__ double
finish_fast64(double * u2, double dx, const PhysParams & P, bool want_dt, bool & bad)
{
  using H = V<DIM>;
  const double sum = u2[H::IA0] + u2[H::IA1];
  if (bits64(sum) != bits64(1.0))
  {
    const double inv = div64(1.0, sum, bad);
    u2[H::IA0] = mul64(u2[H::IA0], inv, bad);
    u2[H::IA1] = mul64(u2[H::IA1], inv, bad);
  }
  u2[H::ID] = u2[H::IAD0] + u2[H::IAD1];
  if (!want_dt)
    return 0.0;
  double        q[H::NQ];
  const double  c = prim_fast64<DIM, true, false, MG>(u2, q, P, bad);
  const Recip64 rdx = recip64(dx, bad);
  double        r = quot64(c + fabs(q[H::QU]), rdx, bad) + quot64(c + fabs(q[H::QV]), rdx, bad);
  if constexpr (DIM == 3)
    r = r + quot64(c + fabs(q[H::QW]), rdx, bad);
  return r;
}

// FP64 cold path: the reference's primitives of a cell whose values leave the
// range of the fast form
template <int DIM>
struct State64
{
  double v[V<DIM>::NV];
};

template <int DIM>
__device__ __noinline__ void
prim_ref64(State64<DIM> u, const PhysParams * P, double * sQ, int stride)
{
  double q[V<DIM>::NQ];
  prim_fp64<DIM>(u.v, q, *P);
  for (int k = 0; k < V<DIM>::NQ; ++k)
    sQ[k * stride] = q[k];
}

// ---------------------------------------------------------------------------
// THINC in the fast form.  The profile's two face values of a cell and
// direction share everything but signs, and few cells need them (volume
// fraction between thinc_eps and 1 - thinc_eps, monotone): the block lists its
// interface (cell, direction) pairs in shared memory and evaluates the list
// with full warps before the faces, which then read the volume fraction (or
// THINC_NONE).  Inline in the face code, the hyperbolic tangents ran in every
// warp that held one interface face and their code made all warps miss the
// instruction cache (29 % of the stalls): 640 us per shock-bubble step (2D,
// 486k cells) against 405 us without THINC.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double
thinc_none64()
{
  return __longlong_as_double(-1LL);
}

// the S of a ring cell one of whose values left the fast form's range: its
// faces take the reference arithmetic (a NaN, so itself out of range)
__device__ __forceinline__ double
bad_cell64()
{
  return __longlong_as_double(-2LL);
}

// whether the cell takes the THINC profile along a direction (its neighbours'
// volume fractions aM, aP): a product of differences of volume fractions
// cannot underflow, so its sign is the differences'
__device__ __forceinline__ bool
thinc_cell64(double a0, double aM, double aP, const PhysParams & P)
{
  const long long b0 = bits64(a0), bM = bits64(aM), bP = bits64(aP);
  return ((bP > b0 && b0 > bM) || (bP < b0 && b0 < bM)) && b0 > bits64(P.thinc_eps) && b0 < bits64(1.0 - P.thinc_eps);
}

// tanh_d with the divisions on the integer pipes
__device__ __forceinline__ double
tanh_fast64(double x, bool & bad)
{
  const double ax = fabs(x);
  double       t = 1.0;
  if (!(ax > 22.0))
  {
    const double y = 2.0 * ax;
    const bool   small = y < 0.34657359027997264;
    const double k = small ? 0.0 : floor(y * 1.4426950408889634 + 0.5);
    const double r = small ? y : (y - k * 0.6931471824645996) - k * -1.904654299957768e-09;
    double       em = expm1_small_d(r);
    if (!small)
      em = ldexp(em + 1.0, (int)k) - 1.0;
    t = div64(em, em + 2.0, bad);
  }
  return x < 0.0 ? -t : t;
}

// the face values of thinc_alpha64 on both sides, nd the normal's component
__device__ __forceinline__ void
thinc_pair64(double a0, double aM, double aP, double nd, const PhysParams & P, double & right, double & left, bool & bad)
{
  const double hb = 0.5 * (P.thinc_beta * nd + 0.01);
  const double Aa = 0.5 * (aP + aM), Bb = 0.5 * (aP - aM);
  const double C = tanh_fast64(hb, bad);
  const double D = tanh_fast64(div64(hb * (a0 - Aa), Bb, bad), bad);
  const double E = div64(D, C, bad);
  right = Aa + div64(Bb * (C + E), 1.0 + D, bad);
  left = Aa + div64(neg64(Bb) * (C - E), 1.0 - D, bad);
}

// |n_d| = |g_d| / |g| of a Youngs normal
__device__ __forceinline__ double
youngs_ratio64(double gd, double g2, bool & bad)
{
  const double nrm = sqrt64(g2, bad);
  return bits64(nrm) > 0 ? fabs(div64(gd, nrm, bad)) : 0.0;
}

// the partial densities and the mixture's S of a face side with THINC volume
// fraction af; hs: the cell's Hancock sources (without their factor 1/2)
struct ThincSide64
{
  double q0, q1, S;
  bool   bad;
};

static __device__ __noinline__ ThincSide64
thinc_side64(double a0, double af, double r0, double r1, double hs0, double hs1, const PhysParams * P)
{
  ThincSide64 s;
  s.bad = false;
  s.q0 = __fma_rn(0.5, hs0, r0 + mul64(div64(r0, a0, s.bad), af - a0, s.bad));
  s.q1 = __fma_rn(0.5, hs1, r1 + mul64(div64(r1, 1.0 - a0, s.bad), a0 - af, s.bad));
  s.S = mix_S64(*P, af, 1.0 - af, s.bad);
  return s;
}

} // namespace g5
