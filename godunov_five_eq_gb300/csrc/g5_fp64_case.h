// g5_fp64_case.h — which form of the FP64 arithmetic a case takes, and the
// grid's SM count (the FP64 translation units).
#pragma once

#include <type_traits>

#include "g5_common.cuh"

namespace g5
{

inline int
num_sms()
{
  static int n = 0;
  if (n == 0)
  {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0)
      n = 1;
  }
  return n;
}

// the FP64 kernels' forms: the fast arithmetic of g5_fast64.cuh for stiffened
// gases and for Mie-Grueneisen laws, and the reference arithmetic as it is
// written for constants outside the fast form's range
constexpr int FAST64 = 0, FASTMG64 = 1, REF64 = 2;

// which form a case takes: the fast ones want their constants zero or far from
// the ends of the double range, and floors whose products stay in it
inline int
case64(const PhysParams & p)
{
  const auto in = [](double x, double lo, double hi) { return x >= lo && x <= hi; };
  const auto zin = [&](double x) { return x == 0.0 || in(x < 0.0 ? -x : x, 1e-200, 1e200); };
  bool       ok = in(p.smallr, 1e-60, 1e60) && in(p.smallc, 1e-100, 1e100);
  for (int k = 0; k < 2; ++k)
  {
    ok = ok && zin(p.xi[k]) && zin(p.gpx[k]) && zin(p.gamma[k]) && zin(p.pinf[k]);
    if (p.eos_kind[k] != EOS_STIFFENED)
    {
      ok = ok && in(p.mg_rho0[k], 1e-60, 1e60);
      for (int j = 0; j < 8; ++j)
        ok = ok && (p.mg[k][j] == 0.0 || in(p.mg[k][j] < 0.0 ? -p.mg[k][j] : p.mg[k][j], 1e-60, 1e60));
    }
  }
  return !ok ? REF64 : (p.mg_any ? FASTMG64 : FAST64);
}

// f(integral constant of the case's form)
template <typename F>
cudaError_t
launch_case64(const PhysParams & p, F f)
{
  switch (case64(p))
  {
    case FAST64: return f(std::integral_constant<int, FAST64>());
    case FASTMG64: return f(std::integral_constant<int, FASTMG64>());
    default: return f(std::integral_constant<int, REF64>());
  }
}

} // namespace g5
