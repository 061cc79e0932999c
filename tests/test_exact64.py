"""The integer-pipe division, square root and product of the FP64 form
(csrc/g5_exact64.h) against the host's IEEE operations, bit for bit."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "godunov_five_eq_gb300", "csrc")

SOURCE = r"""
#include "g5_exact64.h"
#include <cstdio>
#include <random>
using namespace g5;

static std::mt19937_64 gen(20260101);

static double
make(uint64_t e, uint64_t m, uint64_t s)
{
  const uint64_t b = (s << 63) | (e << 52) | (m & 0xFFFFFFFFFFFFFull);
  double         x;
  std::memcpy(&x, &b, 8);
  return x;
}

// mantissas of few bits, long runs of ones, near powers of two, and random
static double
draw(int span)
{
  uint64_t       m = gen();
  const uint64_t mode = gen() & 15;
  if (mode & 1)
    m &= 0xFFFFF;
  if (mode & 2)
    m &= ~0xFFFFFFFFull;
  if (mode & 4)
    m |= 0xFFFFFFFFF0000ull;
  if (mode == 8)
  {
    m = 1ull << (gen() % 52);
    if (gen() & 1)
      m = 0 - m;
  }
  return make(1023 - span + gen() % (2 * span + 1), m, gen() >> 63);
}

static long wrong = 0, refused = 0;

static void
check(const char * what, double got, double want, bool bad, double a, double b)
{
  if (bad)
    ++refused;
  else if (std::memcmp(&got, &want, 8) != 0 && wrong++ < 5)
    std::printf("%s %a %a: %a, not %a\n", what, a, b, got, want);
}

static void
one(double a, double b)
{
  const bool   raw = x64_raw_bad(a) || x64_raw_bad(b);
  bool         bad = raw;
  const double q = div64(a, b, bad);
  check("div", q, a / b, bad, a, b);
  bad = raw;
  const double p = mul64(a, b, bad);
  check("mul", p, a * b, bad, a, b);
  const double x = std::fabs(a);
  bad = x64_raw_bad(x);
  const double s = sqrt64(x, bad);
  check("sqrt", s, std::sqrt(x), bad, x, 0.0);
}

int
main()
{
  for (long i = 0; i < 3000000; ++i)
  {
    const double a = draw(60), b = draw(60);
    one(a, b);
    one(a * (double)(float)b, a); // quotients of few bits
    const double r = (double)(float)a;
    one(r * r, b); // exact roots
    // quotients and roots next to a midpoint
    one(std::nextafter(a * b, 0.0), b);
  }
  if (refused)
    std::printf("%ld refused within the range\n", refused);
  const long in_range = refused;
  for (long i = 0; i < 1000000; ++i)
    one(draw(1000), draw(1000)); // refused or right
  const double special[] = { 0.0, -0.0, 1.0, -1.0, 4.9e-324, 1e-310, 2.2250738585072014e-308, 1e-271, 1.2e-271, 5e210, 6e210, 1.7e308,
                             HUGE_VAL, -HUGE_VAL, std::nan("") };
  for (double a : special)
    for (double b : special)
      one(a, b);
  std::printf("wrong %ld refused in range %ld\n", wrong, in_range);
  return wrong != 0 || in_range != 0;
}
"""


def test_exact64_against_ieee(tmp_path):
    src = tmp_path / "exact64.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "exact64"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    if run.returncode:
        pytest.fail(run.stdout)
