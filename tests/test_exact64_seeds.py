"""The float seeds of the integer-pipe division and square root
(csrc/g5_exact64.h): on the host, seeds as far off as PTX lets rcp.approx
(2^-23 in absolute terms) and rsqrt.approx (2^-22.9 of the value) be, both
ways; on the GPU, every seed the two instructions return, and the operations on
operands of every such mantissa against the hardware's.  Bit for bit."""
import subprocess

import pytest

from godunov_five_eq_gb300 import build

HOST = r"""
#include "g5_exact64.h"
#include <cstdio>
#include <random>
using namespace g5;

static std::mt19937_64 gen(7);

// a float, n units of the last place away
static uint32_t
bits(float f, int n)
{
  uint32_t b;
  std::memcpy(&b, &f, 4);
  return b + n;
}

static double
value(uint32_t b)
{
  float f;
  std::memcpy(&f, &b, 4);
  return f;
}

// mantissas in [1, 2): dense at both ends, the rest random
static double
mantissa()
{
  uint64_t       m = gen() & 0xFFFFFFFFFFFFFull;
  const uint64_t mode = gen() & 3;
  if (mode == 0)
    m >>= 20 + gen() % 20;
  if (mode == 1)
    m |= 0xFFFFFFFFFFFFFull << (12 + gen() % 20) & 0xFFFFFFFFFFFFFull;
  if (mode == 2 && (gen() & 1))
    m = 0xFFFFFFFFFFFFFull - (gen() & 0x3FFFFFFF);
  m |= 1023ull << 52;
  double x;
  std::memcpy(&x, &m, 8);
  return x;
}

static long wrong = 0;

static void
check(const char * what, double got, double want, bool bad, double a, double b, uint32_t seed)
{
  if ((bad || std::memcmp(&got, &want, 8) != 0) && wrong++ < 8)
    std::printf("%s %a %a with seed %08x: %a, not %a\n", what, a, b, seed, got, want);
}

int
main()
{
  const double sq = std::exp2(-22.9);
  for (long i = 0; i < 1000000; ++i)
  {
    const double b = mantissa(), a = mantissa(), x = mantissa() * (1.0 + (gen() & 1));
    const double f = value(x64_float_mant(x64_hi(b), x64_lo(b), 0u));
    for (int n = -5; n <= 5; ++n)
    {
      const uint32_t seed = bits((float)(1.0 / f), n);
      if (std::fabs(value(seed) - 1.0 / f) > 0x1p-23)
        continue;
      bool          bad = false;
      const Recip64 r = recip64_seeded(b, seed, bad);
      check("div", quot64(a, r, bad), a / b, bad, a, b, seed);
      check("div", quot64(b, r, bad), 1.0, bad, b, b, seed);
    }
    const double g = value(x64_float_mant(x64_hi(x), x64_lo(x), x64_odd(x64_hi(x))));
    if (g < 1.0 || g > 4.0)
      return 2;
    for (int n = -5; n <= 5; ++n)
    {
      const uint32_t seed = bits((float)(1.0 / std::sqrt(g)), n);
      if (std::fabs(value(seed) * std::sqrt(g) - 1.0) > sq)
        continue;
      check("sqrt", sqrt64_seeded(x, seed), std::sqrt(x), false, x, 0.0, seed);
    }
  }
  std::printf("wrong %ld\n", wrong);
  return wrong != 0;
}
"""

DEVICE = r"""
#include "g5_exact64.h"
#include <cmath>
#include <cstdio>
using namespace g5;

struct Counts
{
  unsigned long long seeds, rcp_off, rsqrt_off, ops, div_wrong, sqrt_wrong, mul_wrong;
};

__device__ uint64_t
scramble(uint64_t x)
{
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__device__ void
operate(double a, double b, Counts & c)
{
  ++c.ops;
  bool         bad = false;
  const double q = div64(a, b, bad), s = sqrt64(b, bad), p = mul64(a, b, bad);
  c.div_wrong += bad || __double_as_longlong(q) != __double_as_longlong(__ddiv_rn(a, b));
  c.sqrt_wrong += bad || __double_as_longlong(s) != __double_as_longlong(__dsqrt_rn(b));
  c.mul_wrong += bad || __double_as_longlong(p) != __double_as_longlong(__dmul_rn(a, b));
}

// every 24-bit mantissa k 2^-23 of [1, 2] (k = 2^23 .. 2^24) and, doubled, of [2, 4]
__global__ void
all_seeds(Counts * out, double rsqrt_bound)
{
  Counts c = {};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= (1u << 24); i += gridDim.x * blockDim.x)
  {
    const uint32_t fb = 0x3F800000u + i; // [1, 4]
    const double   f = (double)__uint_as_float(fb);
    ++c.seeds;
    if (i <= (1u << 23))
      c.rcp_off += !(fabs((double)__uint_as_float(x64_seed_rcp(fb)) - 1.0 / f) <= 0x1p-23);
    c.rsqrt_off += !(fabs((double)__uint_as_float(x64_seed_rsqrt(fb)) * sqrt(f) - 1.0) <= rsqrt_bound);
    // operands that round to this mantissa: itself, the ends of the interval and between
    const uint64_t m = ((uint64_t)(i & 0x7FFFFFu) << 29);
    for (int k = 0; k < 4; ++k)
    {
      const uint64_t r = scramble((uint64_t)i * 4 + k);
      const int64_t  d = k == 0 ? 0 : (k == 1 ? -0x0FFFFFFF : (k == 2 ? 0x0FFFFFFF : (int64_t)(r & 0x1FFFFFFF) - 0x10000000));
      const uint64_t b = ((uint64_t)(1023u + (i >= (1u << 24) ? 2u : (uint32_t)(i >= (1u << 23)))) << 52) + m + (uint64_t)d;
      const uint64_t a = ((uint64_t)(963u + r % 121u) << 52) | (r >> 12);
      operate(__longlong_as_double((long long)a), __longlong_as_double((long long)b), c);
      // the quotient 1 and the neighbours of 1
      operate(__longlong_as_double((long long)b), __longlong_as_double((long long)b), c);
      operate(__longlong_as_double((long long)b - 1), __longlong_as_double((long long)b), c);
    }
  }
  unsigned long long * o = (unsigned long long *)out, * v = (unsigned long long *)&c;
  for (int k = 0; k < (int)(sizeof(Counts) / 8); ++k)
    atomicAdd(o + k, v[k]);
}

int
main()
{
  Counts * d = nullptr;
  Counts   h = {};
  if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess)
    return 3;
  all_seeds<<<608, 256>>>(d, std::exp2(-22.9));
  if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess)
    return 4;
  std::printf("seeds %llu rcp off %llu rsqrt off %llu operands %llu div wrong %llu sqrt wrong %llu mul wrong %llu\n", h.seeds, h.rcp_off, h.rsqrt_off, h.ops,
              h.div_wrong, h.sqrt_wrong, h.mul_wrong);
  return h.seeds != (1u << 24) + 1u || h.rcp_off || h.rsqrt_off || h.div_wrong || h.sqrt_wrong || h.mul_wrong;
}
"""


def run(cmd, src, exe):
    subprocess.run([*cmd, "-I", build.CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_operations_with_the_least_accurate_seeds(tmp_path):
    src = tmp_path / "seeds.cpp"
    src.write_text(HOST)
    run(["g++", "-O2", "-std=c++17", "-ffp-contract=off"], src, tmp_path / "seeds")


@pytest.mark.gpu
def test_every_seed_of_the_gpu(tmp_path):
    src = tmp_path / "seeds.cu"
    src.write_text(DEVICE)
    run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false"], src, tmp_path / "seeds")
