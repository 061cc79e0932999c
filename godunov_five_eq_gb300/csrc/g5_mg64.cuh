// g5_mg64.cuh — the Mie-Grueneisen mixture rules of the FP64 form (mg_law,
// mg_mixture, mg_bulk_modulus in g5_common.cuh) from the operations of
// g5_exact64.h: same expressions, same order, same doubles.
//
// A mixture evaluation in hardware FP64 is about a dozen divisions (4.5 clocks
// each per SM) besides the two exponentials' Horner chains, nine times per
// cell and step.  Here the divisions run on the integer pipes, each divisor's
// quotients share its reciprocal, half of the Horner products run there too,
// and a stiffened-gas material (whose law is a constant) costs three products.
// The functions are calls: inlined at each use they would not fit the
// instruction cache.  The two shock-wave laws keep their hardware arithmetic
// (mg_law), with the range tests.
#pragma once

#include "g5_common.cuh"
#include "g5_exact64.h"

namespace g5
{

struct Law64
{
  double G, dG, f, df;
  bool   bad;
};

struct Mix64
{
  double S, PI, C1, C0; // p S = rho e - PI, rho c^2 S = p C1 + C0
};

struct MixBad64
{
  Mix64 m;
  bool  bad;
};

// exp_d for x in its normal-result range, else bad
__device__ __forceinline__ double
exp_fast64(double x, bool & bad)
{
  const double k = floor(x * 1.4426950408889634 + 0.5);
  const double r = (x - k * 0.6931471824645996) - k * -1.904654299957768e-09;
  const double e = expm1_small_d(r) + 1.0; // in [0.7, 1.5]
  const int    n = (int)k;
  bad = bad || n < -890 || n > 690; // (the range of g5_exact64.h)
  return x64_make(x64_hi(e) + ((uint32_t)n << 20), x64_lo(e));
}

static __device__ __noinline__ Law64
mg_law_fast64(const PhysParams * P, int k, double rho)
{
  Law64 L;
  L.bad = x64_raw_bad(rho);
  if (P->eos_kind[k] == EOS_JWL)
  {
    const double * c = P->mg[k];
    const double   rho0 = c[0], w = c[1], A1 = c[2], A2 = c[3], R1 = c[4], R2 = c[5], e0 = c[6];
    const Recip64  ir = recip64(rho, L.bad);
    const double   x1 = quot64(R1 * rho0, ir, L.bad), x2 = quot64(R2 * rho0, ir, L.bad);
    const double   w1 = div64(w, x1, L.bad), w2 = div64(w, x2, L.bad);
    const double   E1 = exp_fast64(-x1, L.bad), E2 = exp_fast64(-x2, L.bad);
    // (f multiplies A (1 - w/x) first, f' A E)
    const double F1 = mul64(mul64(A1, 1.0 - w1, L.bad), E1, L.bad), F2 = mul64(mul64(A2, 1.0 - w2, L.bad), E2, L.bad);
    const double H1 = mul64(mul64(A1, E1, L.bad), x1 - w - w1, L.bad), H2 = mul64(mul64(A2, E2, L.bad), x2 - w - w2, L.bad);
    L.G = w;
    L.dG = 0.0;
    L.f = (F1 + F2) - mul64(mul64(w, rho, L.bad), e0, L.bad);
    L.df = quot64(H1 + H2, ir, L.bad) - w * e0;
  }
  else
  {
    mg_law(*P, k, rho, L.G, L.dG, L.f, L.df);
    L.bad = L.bad || x64_raw_bad(L.G) || x64_raw_bad(L.dG) || x64_raw_bad(L.f) || x64_raw_bad(L.df);
  }
  return L;
}

__device__ __forceinline__ double
mg_density_fast64(const PhysParams * P, int k, double a, double ar, bool & bad)
{
  if (!(__double_as_longlong(a) > 0))
    return P->mg_rho0[k];
  const double r = div64(ar, a, bad);
  return __double_as_longlong(r) > __double_as_longlong(P->smallr) ? r : P->smallr;
}

// mg_mixture: each sum starts from 0, material 0 first
static __device__ __noinline__ MixBad64
mg_mixture_fast64(const PhysParams * P, double a0, double a1, double ar0, double ar1)
{
  MixBad64 r;
  r.bad = false;
  double S = 0.0, PI = 0.0, C1 = 0.0, C0 = 0.0;
#pragma unroll 1
  for (int k = 0; k < 2; ++k)
  {
    const double a = k == 0 ? a0 : a1;
    if (P->eos_kind[k] == EOS_STIFFENED)
    {
      // G' = f' = 0: h = xi, and f = -gamma pinf
      const double xi = P->xi[k], ax = mul64(a, xi, r.bad);
      S = S + ax;
      C1 = C1 + mul64(a, xi + 1.0, r.bad);
      if (P->pi64 & (1 << k))
      {
        const double gp = P->gamma[k] * P->pinf[k];
        PI = PI + mul64(ax, gp, r.bad);
        C0 = C0 + mul64(a, mul64(xi, gp, r.bad), r.bad);
      }
      continue;
    }
    const double rho = mg_density_fast64(P, k, a, k == 0 ? ar0 : ar1, r.bad);
    const Law64  L = mg_law_fast64(P, k, rho);
    r.bad = r.bad || L.bad;
    const double xi = div64(1.0, L.G, r.bad);
    const double h = mul64(xi, 1.0 + mul64(mul64(rho, L.dG, r.bad), xi, r.bad), r.bad);
    const double ax = mul64(a, xi, r.bad);
    S = S + ax;
    PI = PI - mul64(ax, L.f, r.bad);
    C1 = C1 + mul64(a, h + 1.0, r.bad);
    C0 = C0 + mul64(a, mul64(mul64(xi, rho, r.bad), L.df, r.bad) - mul64(h, L.f, r.bad), r.bad);
  }
  r.m.S = S;
  r.m.PI = PI;
  r.m.C1 = C1;
  r.m.C0 = C0;
  return r;
}

} // namespace g5
