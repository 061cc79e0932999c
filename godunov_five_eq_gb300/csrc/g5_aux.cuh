// g5_aux.cuh — boundary fill of outside blocks, standalone CFL reduction,
// refine flags and the device-side dt update of the solver loop.
#pragma once

#include <type_traits>

#include "g5_common.cuh"
#include "g5_fast64.cuh"

namespace g5
{

// FillOutsideCellFunctor::operator() (border_conditions/FillOutside.cpp:71-170):
// one thread per outside cell.  The reference visits the faces in order and
// every face that applies rewrites the whole cell, so the last such face
// wins: it is found first (from the outside block's row, read in one wave),
// then the cell is copied once.
template <int DIM, int B>
__global__ void
fill_outside_kernel(double * U, DevMesh m, PhysParams P)
{
  using H = V<DIM>;
  constexpr int NC = (DIM == 2) ? B * B : B * B * B;
  const long    gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long)m.n_outside * NC)
    return;
  const int o = (int)(gid / NC), c = (int)(gid % NC);
  const int nout = m.n_owned + o;
  const int nin = m.out_src[o];
  int8_t    border[6], normal[3];
#pragma unroll
  for (int f = 0; f < 2 * DIM; ++f)
    border[f] = m.out_border[o * 6 + f];
#pragma unroll
  for (int e = 0; e < DIM; ++e)
    normal[e] = m.out_normal[o * 3 + e];
  if (nin < 0 || nin >= m.n_owned)
    return;
  int last = -1;
#pragma unroll
  for (int face = 0; face < 2 * DIM; ++face)
    if (border[face] && normal[face >> 1] != 0 && (P.bc[face] == 2 || P.bc[face] == 3))
      last = face;
  if (last < 0)
    return;
  const int dir = last >> 1, bc = P.bc[last];
  int       ci[3] = { c % B, (c / B) % B, DIM == 3 ? c / (B * B) : 0 };
  ci[dir] = bc == 2 ? ((last & 1) ? B - 1 : 0) : B - 1 - ci[dir];
  const int      cin = ci[0] + B * (ci[1] + B * ci[2]);
  const double * src = U + (size_t)nin * H::NV * NC + cin;
  double *       dst = U + (size_t)nout * H::NV * NC + c;
  double         u[H::NV];
#pragma unroll
  for (int v = 0; v < H::NV; ++v)
    u[v] = src[v * NC];
  if (bc == 3)
    u[H::IU + dir] = -u[H::IU + dir];
#pragma unroll
  for (int v = 0; v < H::NV; ++v)
    dst[v * NC] = u[v];
}

// CFL rate of one cell (ComputeDtFiveEqFunctor.cpp:87-134) in the reference's
// arithmetic (KIND 2), and from the fast operations of g5_fast64.cuh (KIND 0
// stiffened gases, 1 Mie-Grueneisen laws)
template <int DIM>
__device__ __forceinline__ double
cfl_rate_ref64(const double * u, double dx, const PhysParams & P)
{
  using H = V<DIM>;
  double       q[H::NQ];
  const double cs = prim_fp64<DIM>(u, q, P);
  double       r = (cs + fabs(q[H::QU])) / dx + (cs + fabs(q[H::QV])) / dx;
  if constexpr (DIM == 3)
    r = r + (cs + fabs(q[H::QW])) / dx;
  return r;
}

template <int DIM>
__device__ __noinline__ double
cfl_rate_cold64(State64<DIM> s, double dx, const PhysParams * P)
{
  return cfl_rate_ref64<DIM>(s.v, dx, *P);
}

template <int DIM, int KIND>
__device__ __forceinline__ double
cfl_rate64(const double * u, double dx, const PhysParams & P)
{
  using H = V<DIM>;
  if constexpr (KIND == 2)
    return cfl_rate_ref64<DIM>(u, dx, P);
  else
  {
    double        q[H::NQ];
    bool          bad = x64_raw_bad(dx);
    const double  c = prim_fast64<DIM, true, true, KIND == 1>(u, q, P, bad);
    const Recip64 rdx = recip64(dx, bad);
    double        r = quot64(c + fabs(q[H::QU]), rdx, bad) + quot64(c + fabs(q[H::QV]), rdx, bad);
    if constexpr (DIM == 3)
      r = r + quot64(c + fabs(q[H::QW]), rdx, bad);
    if (bad)
    {
      State64<DIM> s;
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
        s.v[v] = u[v];
      r = cfl_rate_cold64<DIM>(s, dx, &P);
    }
    return r;
  }
}

// max over the block of the threads' rates into the instance's accumulator
// (sred: one value per warp; every thread of the CTA calls it)
__device__ __forceinline__ void
block_max_rate64(double mx, double * sred, double * acc)
{
  mx = warp_max_pos64(mx);
  if ((threadIdx.x & 31) == 0)
    sred[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    double mm = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
      mm = bits64(sred[w]) > bits64(mm) ? sred[w] : mm;
    atomic_max_pos(acc, mm);
  }
  __syncthreads();
}

// larger of a running rate (>= 0) and a cell's (NaN and negative ones do not count)
__device__ __forceinline__ double
max_rate64(double mx, double r)
{
  const long long b = bits64(r);
  return b > bits64(mx) && b <= 0x7FF0000000000000LL ? r : mx;
}

// ComputeDtFiveEqFunctor: one CTA per block, block max, one atomic per CTA
template <int DIM, int B, int KIND>
__global__ void __launch_bounds__(256)
inv_dt_kernel(const double * U, DevMesh m, const __grid_constant__ PhysParams P, double * invdt)
{
  using H = V<DIM>;
  constexpr int NC = (DIM == 2) ? B * B : B * B * B;
  __shared__ double sred[32];
  for (int n = blockIdx.x; n < m.n_owned; n += gridDim.x)
  {
    const double dx = P.level_dx[m.level[n]];
    double       mx = 0.0;
    for (int c = threadIdx.x; c < NC; c += blockDim.x)
    {
      double u[H::NV];
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
        u[v] = U[((size_t)n * H::NV + v) * NC + c];
      mx = max_rate64(mx, cfl_rate64<DIM, KIND>(u, dx, P));
    }
    block_max_rate64(mx, sred, invdt + (m.inst ? m.inst[n] : 0));
  }
}

// RK2_SSP final stage (SolverGodunovFiveEq.cpp:519-520, the external
// LinearCombination with the SSP coefficients): U2 = 0.5 U + 0.5 U2 on the
// owned blocks, fused with the CFL rate of the result (one CTA per block).
template <int DIM, int B, bool MIXED, int KIND = 2>
__global__ void __launch_bounds__(256)
rk2_combine_kernel(const double * U, double * U2, DevMesh m, const __grid_constant__ PhysParams P, double * invdt)
{
  using H = V<DIM>;
  constexpr int NC = (DIM == 2) ? B * B : B * B * B;
  using DtT = typename std::conditional<MIXED, float, double>::type;
  __shared__ DtT sred[32];
  const int      eosk = P.mg_any ? 2 : ((P.gpx[0] != 0.0 || P.gpx[1] != 0.0) ? 1 : 0);
  for (int n = blockIdx.x; n < m.n_owned; n += gridDim.x)
  {
    const double dx = P.level_dx[m.level[n]];
    DtT          mx = DtT(0);
    for (int c = threadIdx.x; c < NC; c += blockDim.x)
    {
      double u[H::NV];
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
      {
        const size_t i = ((size_t)n * H::NV + v) * NC + c;
        u[v] = 0.5 * U[i] + 0.5 * U2[i];
        U2[i] = u[v];
      }
      if constexpr (MIXED)
      {
        float       d, ux, uy, uz, a0;
        const float p = pressure_mixed<DIM>(u, P, eosk, d, ux, uy, uz, a0);
        const float cs = sound_speed_eos(P, eosk, d, p, fmaxf(0.0f, fminf(1.0f, a0)), d2f_fast(u[H::IAD0]), d2f_fast(u[H::IAD1]));
        float       r = (cs + fabsf(ux)) + (cs + fabsf(uy));
        if constexpr (DIM == 3)
          r += cs + fabsf(uz);
        mx = fmaxf(mx, r * __frcp_rn(d2f_fast(dx)));
      }
      else if (invdt)
        mx = max_rate64(mx, cfl_rate64<DIM, KIND>(u, dx, P));
    }
    if constexpr (!MIXED)
    {
      if (invdt)
        block_max_rate64(mx, sred, invdt + (m.inst ? m.inst[n] : 0));
    }
    else if (invdt)
    {
      for (int o = 16; o > 0; o >>= 1)
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if ((threadIdx.x & 31) == 0)
        sred[threadIdx.x >> 5] = mx;
      __syncthreads();
      if (threadIdx.x == 0)
      {
        DtT mm = DtT(0);
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
          mm = fmax(mm, sred[w]);
        atomic_max_pos(invdt + (m.inst ? m.inst[n] : 0), (double)mm);
      }
    }
    __syncthreads();
  }
}

// dt = cfl / inv_dt per instance; inv_dt accumulator cleared for the next step
static __global__ void
dt_update_kernel(double * invdt, double * dt, double * dt_hist, int n_inst, double cfl)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_inst)
    return;
  const double d = cfl / invdt[i];
  dt[i] = d;
  if (dt_hist)
    dt_hist[i] = d;
  invdt[i] = 0.0;
}

// ComputeRefineFlags (scheme/ComputeRefineFlags.cpp:66-368): value of the
// same-level face neighbour of a cell (getNeighborDataSameLevel)
template <int DIM, int B>
__device__ double
neighbor_same_level(const double * U, const DevMesh & m, int n, const int * cell, int dir, int side, int var)
{
  using H = V<DIM>;
  constexpr int NC = (DIM == 2) ? B * B : B * B * B;
  constexpr int NS = (DIM == 2) ? 9 : 27, NCH = (DIM == 2) ? 4 : 8;
  auto          cidx = [](int x, int y, int z) { return x + B * (y + B * z); };
  int           g[3] = { cell[0], cell[1], cell[2] };
  g[dir] += side;
  if (g[dir] >= 0 && g[dir] < B)
    return U[((size_t)n * H::NV + var) * NC + cidx(g[0], g[1], g[2])];
  int d[3] = { 0, 0, 0 }, v[3] = { g[0], g[1], g[2] };
  d[dir] = side;
  v[dir] = g[dir] - side * B;
  const int s = (d[0] + 1) + 3 * (d[1] + 1) + (DIM == 3 ? 9 * (d[2] + 1) : 0);
  const int rel = m.nbr_rel[n * NS + s];
  const int * nb = m.nbr + (n * NS + s) * NCH;
  const double here = U[((size_t)n * H::NV + var) * NC + cidx(cell[0], cell[1], cell[2])];
  if (rel <= 0)
  {
    const int src = nb[0];
    if (src < 0 || src >= m.n_owned)
      return here; // outside the domain: value of the current cell
    if (rel == 0)
      return U[((size_t)src * H::NV + var) * NC + cidx(v[0], v[1], v[2])];
    int cc[3] = { 0, 0, 0 };
    for (int e = 0; e < DIM; ++e)
      cc[e] = ((m.coord[n * 3 + e] + d[e]) & 1) * (B / 2) + (v[e] >> 1);
    return U[((size_t)src * H::NV + var) * NC + cidx(cc[0], cc[1], cc[2])];
  }
  int f0[3] = { 0, 0, 0 }, ch[3] = { 0, 0, 0 };
  for (int e = 0; e < DIM; ++e)
  {
    const int f = 2 * v[e];
    ch[e] = f / B;
    f0[e] = f - ch[e] * B;
  }
  const int F = nb[ch[0] + 2 * ch[1] + 4 * ch[2]];
  if (F < 0 || F >= m.n_owned)
    return here;
  double sum = 0.0;
  for (int oz = 0; oz < (DIM == 3 ? 2 : 1); ++oz)
    for (int oy = 0; oy < 2; ++oy)
      for (int ox = 0; ox < 2; ++ox)
        sum += U[((size_t)F * H::NV + var) * NC + cidx(f0[0] + ox, f0[1] + oy, f0[2] + oz)];
  return sum / (double)(1 << DIM);
}

__device__ __forceinline__ double
normalized_gradient(double v1, double v2)
{
  double vmax = fmax(fabs(v1), fabs(v2));
  if (vmax < 0.001)
    return 0.0;
  vmax = fabs(v1 - v2) / vmax;
  return fmax(fmin(vmax, 1.0), 0.0);
}

template <int DIM, int B>
__global__ void
refine_flags_kernel(const double * U,
                    DevMesh        m,
                    int            indicator,
                    double         eps_r,
                    double         eps_c,
                    double         eps_l,
                    int            lmin,
                    int            lmax,
                    int8_t *       flags)
{
  using H = V<DIM>;
  constexpr int NC = (DIM == 2) ? B * B : B * B * B;
  __shared__ int sflag;
  for (int n = blockIdx.x; n < m.n_owned; n += gridDim.x)
  {
    if (threadIdx.x == 0)
      sflag = -1;
    __syncthreads();
    const int lev = m.level[n];
    int       bflag = -1;
    for (int c = threadIdx.x; c < NC; c += blockDim.x)
    {
      const int cell[3] = { c % B, (c / B) % B, DIM == 3 ? c / (B * B) : 0 };
      int       flag = -1;
      auto      update = [&](double ind) {
        int f;
        if (lev < lmax && ind > eps_r)
          f = 2;
        else if (lev > lmin && ind < eps_c)
          f = 0;
        else
          f = 1;
        flag = flag > f ? flag : f;
      };
      const int vars[2] = { H::IAD0, H::IAD1 };
      if (indicator == 2)
      {
        for (int t = 0; t < 2; ++t)
          for (int d = 0; d < DIM; ++d)
          {
            const double L = neighbor_same_level<DIM, B>(U, m, n, cell, d, -1, vars[t]);
            const double R = neighbor_same_level<DIM, B>(U, m, n, cell, d, +1, vars[t]);
            const double C = U[((size_t)n * H::NV + vars[t]) * NC + c];
            update(fabs(L - 2 * C + R) / (fabs(R - C) + fabs(C - L) + eps_l * (fabs(L) + 2 * fabs(C) + fabs(R))));
          }
      }
      else
      {
        for (int t = 0; t < 2; ++t)
        {
          const double C = U[((size_t)n * H::NV + vars[t]) * NC + c];
          if (indicator == 1)
          {
            double num = 0.0, den = 0.0;
            for (int d = 0; d < DIM; ++d)
            {
              const double L = neighbor_same_level<DIM, B>(U, m, n, cell, d, -1, vars[t]);
              const double R = neighbor_same_level<DIM, B>(U, m, n, cell, d, +1, vars[t]);
              const double aa = L - 2 * C + R;
              num = d == 0 ? aa * aa : num + aa * aa;
              const double tmp = fabs(R - C) + fabs(C - L) + eps_l * (fabs(L) + 2 * fabs(C) + fabs(R));
              den = d == 0 ? tmp * tmp : den + tmp * tmp;
            }
            update(sqrt(num / den));
          }
          else
          {
            double res = -1.7976931348623157e308;
            for (int d = 0; d < DIM; ++d)
            {
              const double L = neighbor_same_level<DIM, B>(U, m, n, cell, d, -1, vars[t]);
              const double R = neighbor_same_level<DIM, B>(U, m, n, cell, d, +1, vars[t]);
              res = fmax(res, normalized_gradient(C, L));
              res = fmax(res, normalized_gradient(C, R));
            }
            update(res);
          }
        }
      }
      bflag = bflag > flag ? bflag : flag;
    }
    atomicMax(&sflag, bflag);
    __syncthreads();
    if (threadIdx.x == 0)
      flags[n] = (int8_t)sflag;
    __syncthreads();
  }
}

// The SIMPLE_GRADIENT indicator (normalized_gradient of every face pair of
// both partial densities) without its divisions.  A block's flag needs only
// its largest indicator, compared with eps_r and eps_c: it is found in FP32
// (the differences in FP64, everything else on floats), and only a block
// whose largest indicator lies within 1e-5 of a threshold, or that holds
// values floats do not decide (infinities, NaN, magnitudes of 1e30 and more or
// at the reference's 0.001), evaluates the reference's rounded quotients.
// Every interior pair is taken once, from a shared-memory copy of the block.
// One thread per cell.  2.0M cells: the division form was bound by the FP64
// pipe (24 divisions per cell, 732 us), a form comparing every pair with both
// thresholds by the ALU pipe (980 instructions per cell, 94 us).
template <int DIM, int B>
struct GradientTile
{
  static constexpr int NC = DIM == 2 ? B * B : B * B * B, NF = 2 * DIM, FC = NC / B;
  double v[2][NC], h[2][NF * FC]; // the block, its face neighbours
  float  vf[2][NC], hf[2][NF * FC];
};

// neighbor_same_level of both partial densities for a cell on the block's face
template <int DIM, int B>
__device__ __forceinline__ void
halo_densities(const double * __restrict__ U, const DevMesh & m, int n, const int * cell, int dir, int side, double & h0, double & h1)
{
  using H = V<DIM>;
  constexpr int NC = (DIM == 2) ? B * B : B * B * B;
  constexpr int NS = (DIM == 2) ? 9 : 27, NCH = (DIM == 2) ? 4 : 8;
  const int     s = NS / 2 + side * (dir == 0 ? 1 : (dir == 1 ? 3 : 9));
  const int     rel = m.nbr_rel[n * NS + s];
  const int *   nb = m.nbr + (n * NS + s) * NCH;
  int           v[3] = { cell[0], cell[1], cell[2] };
  v[dir] = side < 0 ? B - 1 : 0; // the same-level neighbour's cell
  int c[3] = { v[0], v[1], v[2] }, src = nb[0];
  if (rel < 0)
  {
#pragma unroll
    for (int e = 0; e < DIM; ++e)
      c[e] = ((m.coord[n * 3 + e] + (e == dir ? side : 0)) & 1) * (B / 2) + (v[e] >> 1);
  }
  else if (rel > 0)
  {
    int kid = 0;
#pragma unroll
    for (int e = 0; e < DIM; ++e)
    {
      const int k = v[e] >= B / 2 ? 1 : 0;
      kid |= k << e;
      c[e] = 2 * v[e] - k * B;
    }
    src = nb[kid];
  }
  const bool here = src < 0 || src >= m.n_owned; // outside the domain: the cell itself
  const int  k = here ? cell[0] + B * (cell[1] + B * cell[2]) : c[0] + B * (c[1] + B * c[2]);
  const double * p = U + (size_t)(here ? n : src) * H::NV * NC + k;
  if (here || rel <= 0)
  {
    h0 = p[H::IAD0 * NC];
    h1 = p[H::IAD1 * NC];
    return;
  }
  h0 = 0.0;
  h1 = 0.0;
#pragma unroll
  for (int o = 0; o < NCH; ++o)
  {
    const int off = (o & 1) + B * (((o >> 1) & 1) + B * (o >> 2));
    h0 += p[H::IAD0 * NC + off];
    h1 += p[H::IAD1 * NC + off];
  }
  h0 = h0 / NCH;
  h1 = h1 / NCH;
}

// f(variable, own value's index, neighbour's index or -1 - halo index) over the
// face pairs of one cell
template <int DIM, int B, typename F>
__device__ __forceinline__ void
gradient_pairs(int tid, F f)
{
  constexpr int FC = GradientTile<DIM, B>::FC;
  const int     cell[3] = { tid % B, (tid / B) % B, DIM == 3 ? tid / (B * B) : 0 };
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int d = 0; d < DIM; ++d)
    {
      const int o = d == 0 ? 1 : (d == 1 ? B : B * B);
      const int p = d == 0 ? cell[1] + (DIM == 3 ? B * cell[2] : 0) : (d == 1 ? cell[0] + (DIM == 3 ? B * cell[2] : 0) : cell[0] + B * cell[1]);
      f(t, cell[d] < B - 1 ? tid + o : -1 - ((2 * d + 1) * FC + p));
      if (cell[d] == 0)
        f(t, -1 - (2 * d * FC + p));
    }
}

// the cell's pairs in the reference's arithmetic: bit 0 some indicator above
// eps_r, bit 1 some not below eps_c
template <int DIM, int B>
__device__ __noinline__ int
gradient_exact(const GradientTile<DIM, B> * g, int tid, double eps_r, double eps_c)
{
  int bits = 0;
  gradient_pairs<DIM, B>(tid, [&](int t, int n) {
    const double ind = normalized_gradient(g->v[t][tid], n >= 0 ? g->v[t][n] : g->h[t][-1 - n]);
    bits |= (ind > eps_r ? 1 : 0) | (ind < eps_c ? 0 : 2);
  });
  return bits;
}

template <int DIM, int B>
__global__ void __launch_bounds__(DIM == 2 ? B * B : B * B * B)
gradient_flags_kernel(const double * __restrict__ U, DevMesh m, double eps_r, double eps_c, float rf, float cf, int lmin, int lmax, int8_t * flags)
{
  using H = V<DIM>;
  using T = GradientTile<DIM, B>;
  constexpr int NC = T::NC, NF = T::NF, FC = T::FC;
  __shared__ T        g;
  __shared__ unsigned sMax[2]; // largest indicator (float bits; all ones: undecided) of this and the next block
  const int           tid = threadIdx.x;
  if (tid < 2)
    sMax[tid] = 0u;
  int par = 0;
  for (int n = blockIdx.x; n < m.n_owned; n += gridDim.x, par ^= 1)
  {
    const int      lev = m.level[n];
    const double * base = U + (size_t)n * H::NV * NC;
    const double   v0 = base[H::IAD0 * NC + tid], v1 = base[H::IAD1 * NC + tid];
    g.v[0][tid] = v0;
    g.v[1][tid] = v1;
    g.vf[0][tid] = fabsf(d2f_nan(v0));
    g.vf[1][tid] = fabsf(d2f_nan(v1));
    for (int h = tid; h < NF * FC; h += NC)
    {
      const int f = h / FC, p = h % FC, dir = f >> 1;
      int       hc[3] = { 0, 0, 0 };
      const int e1 = dir == 0 ? 1 : 0, e2 = dir == 2 ? 1 : 2;
      hc[dir] = (f & 1) ? B - 1 : 0;
      hc[e1] = p % B;
      if (DIM == 3)
        hc[e2] = p / B;
      double h0, h1;
      halo_densities<DIM, B>(U, m, n, hc, dir, (f & 1) ? 1 : -1, h0, h1);
      g.h[0][h] = h0;
      g.h[1][h] = h1;
      g.hf[0][h] = fabsf(d2f_nan(h0));
      g.hf[1][h] = fabsf(d2f_nan(h1));
    }
    __syncthreads();
    float qmax = 0.0f;
    bool  plain = true;
    gradient_pairs<DIM, B>(tid, [&](int t, int k) {
      const double N = k >= 0 ? g.v[t][k] : g.h[t][-1 - k];
      const float  vmax = fmaxf(g.vf[t][tid], k >= 0 ? g.vf[t][k] : g.hf[t][-1 - k]);
      const float  q = __fdividef(fabsf(d2f_fast(g.v[t][tid] - N)), vmax);
      // (a NaN drops out of fmaxf: the sum below keeps it)
      plain = plain && (g.vf[t][tid] + vmax) < 1e30f && fabsf(vmax - 0.001f) > 1e-8f && (k >= 0 ? g.vf[t][k] : g.hf[t][-1 - k]) < 1e30f;
      qmax = fmaxf(qmax, vmax < 0.001f ? 0.0f : q);
    });
    const unsigned w = __reduce_max_sync(0xffffffffu, plain ? __float_as_uint(qmax) : 0xffffffffu);
    if ((tid & 31) == 0)
      atomicMax(&sMax[par], w);
    __syncthreads();
    const unsigned top = sMax[par];
    const float    q = __uint_as_float(top);
    // thresholds of 1 and more decide without the cells (the indicator is at
    // most 1); the others when q is not within 1e-5 of them
    const bool want_r = bits64(eps_r) < bits64(1.0), want_c = bits64(eps_c) <= bits64(1.0);
    bool       above = want_r && q > rf, below = !want_c || q < cf || (q == 0.0f && bits64(eps_c) > 0);
    const bool near = top == 0xffffffffu || (want_r && fabsf(q - rf) <= 1e-5f * rf && q != 0.0f) || (want_c && fabsf(q - cf) <= 1e-5f * cf && q != 0.0f);
    if (near)
    {
      const int x = gradient_exact<DIM, B>(&g, tid, eps_r, eps_c);
      above = __syncthreads_or(x & 1) != 0;
      below = __syncthreads_or(x & 2) == 0;
    }
    if (tid == 0)
    {
      flags[n] = (int8_t)(lev < lmax && above ? 2 : (lev > lmin && below ? 0 : 1));
      sMax[par ^ 1] = 0u; // (last read before the barrier above)
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// block remap after a mesh adaptation (SolverGodunovFiveEq::
// map_userdata_after_adapt, SolverGodunovFiveEq.cpp:1137-1169): one CTA per new
// owned block.  kind 0 copies an old block, kind 1 is the SIMPLE_COPY
// prolongation of one child of an old block (every fine cell takes the parent
// cell containing its centre), kind 2 the restriction of 2^dim old children
// (get_conservative_vars_restriction, ConvertToPrimitivesVariablesFunctor.cpp:
// 208-246: mean of the fine cells for IE IU IV (IW) IAD0 IAD1 IA0, summed in
// z, y, x order, IA1 = 1 - IA0, ID = IAD0 + IAD1).  The host validated kind and
// src, so every index read here is in range.
// ---------------------------------------------------------------------------
template <int DIM, int B>
__global__ void __launch_bounds__(256)
remap_kernel(const double * __restrict__ Uold, double * __restrict__ Unew, const int8_t * __restrict__ kind,
             const int32_t * __restrict__ src, int n_new)
{
  using H = V<DIM>;
  constexpr int NC = DIM == 2 ? B * B : B * B * B;
  constexpr int NCH = 1 << DIM;
  for (int j = blockIdx.x; j < n_new; j += gridDim.x)
  {
    const int       k = kind[j];
    const int32_t * s = src + (size_t)j * NCH;
    double *        out = Unew + (size_t)j * H::NV * NC;
    if (k == 0)
    {
      const double2 * in2 = reinterpret_cast<const double2 *>(Uold + (size_t)s[0] * H::NV * NC);
      double2 *       out2 = reinterpret_cast<double2 *>(out);
      for (int t = threadIdx.x; t < H::NV * NC / 2; t += blockDim.x)
        out2[t] = in2[t];
      continue;
    }
    for (int c = threadIdx.x; c < NC; c += blockDim.x)
    {
      const int cc[3] = { c % B, (c / B) % B, DIM == 3 ? c / (B * B) : 0 };
      if (k == 1)
      {
        const int      ch = s[1];
        const int      px = (ch & 1) * (B / 2) + (cc[0] >> 1);
        const int      py = ((ch >> 1) & 1) * (B / 2) + (cc[1] >> 1);
        const int      pz = DIM == 3 ? ((ch >> 2) & 1) * (B / 2) + (cc[2] >> 1) : 0;
        const double * in = Uold + (size_t)s[0] * H::NV * NC + px + B * (py + B * pz);
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          out[v * NC + c] = in[v * NC];
      }
      else
      {
        int ch[3] = { 0, 0, 0 }, f0[3] = { 0, 0, 0 };
#pragma unroll
        for (int e = 0; e < DIM; ++e)
        {
          const int f = 2 * cc[e];
          ch[e] = f / B;
          f0[e] = f - ch[e] * B;
        }
        const double * in = Uold + (size_t)s[ch[0] + 2 * ch[1] + 4 * ch[2]] * H::NV * NC;
        const int      vars[7] = { H::IE, H::IU, H::IV, H::IW, H::IAD0, H::IAD1, H::IA0 };
#pragma unroll
        for (int t = 0; t < 7; ++t)
        {
          if (DIM == 2 && t == 3)
            continue;
          const int v = vars[t];
          double    sum = 0.0;
#pragma unroll
          for (int oz = 0; oz < (DIM == 3 ? 2 : 1); ++oz)
#pragma unroll
            for (int oy = 0; oy < 2; ++oy)
#pragma unroll
              for (int ox = 0; ox < 2; ++ox)
                sum += in[v * NC + (f0[0] + ox) + B * ((f0[1] + oy) + B * (DIM == 3 ? f0[2] + oz : 0))];
          out[v * NC + c] = sum / (double)(1 << DIM);
        }
        out[H::IA1 * NC + c] = 1.0 - out[H::IA0 * NC + c];
        out[H::ID * NC + c] = out[H::IAD0 * NC + c] + out[H::IAD1 * NC + c];
      }
    }
  }
}

// per-record rows of DeferInfo<DIM> for the records listed in `codes` (one
// thread per record): everything the reflux pass needs before its data loads
template <int DIM>
__global__ void
defer_info_kernel(DevMesh m, const int32_t * codes, int n, int32_t * info)
{
  using D = DeferInfo<DIM>;
  constexpr int NF = 2 * DIM, NS = DIM == 2 ? 9 : 27, NCH = 1 << DIM;
  const int     r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n)
    return;
  const int code = codes[r];
  const int nb = code >> 3;
  int32_t * row = info + (size_t)r * D::STRIDE;
  row[0] = code;
  for (int f = 0; f < NF; ++f)
  {
    const int ds = m.defer_slot[nb * NF + f];
    row[1 + f] = ds;
    const int dir = f >> 1, side = f & 1;
    int       d[3] = { 0, 0, 0 };
    d[dir] = side ? 1 : -1;
    const int s = (d[0] + 1) + 3 * (d[1] + 1) + (DIM == 3 ? 9 * (d[2] + 1) : 0);
    for (int c = 0; c < D::NCF; ++c)
    {
      int rs = -1;
      if (ds >= 0)
      {
        int ch[3] = { 0, 0, 0 };
        ch[dir] = side ? 0 : 1;
        const int e1 = dir == 0 ? 1 : 0, e2 = dir == 2 ? 1 : 2;
        ch[e1] = c & 1;
        if (DIM == 3)
          ch[e2] = c >> 1;
        const int F = m.nbr[((size_t)nb * NS + s) * NCH + ch[0] + 2 * ch[1] + 4 * ch[2]];
        rs = (F >= 0 && F < m.n_owned) ? m.reflux_slot[F * NF + (f ^ 1)] : -1;
      }
      row[D::RS + f * D::NCF + c] = rs;
    }
  }
  row[D::LEVEL] = m.level[nb];
  row[D::INST] = m.inst ? m.inst[nb] : 0;
  for (int k = D::INST + 1; k < D::STRIDE; ++k)
    row[k] = 0;
}

// the derived quantities a field list asks for (bits of FieldList::need)
constexpr int NEED_PRESSURE = 1 << 1, NEED_SOUND = 1 << 2, NEED_EKIN = 1 << 3, NEED_MACH = 1 << 4, NEED_VELOCITY = (1 << 5) | (1 << 6) | (1 << 7);

// ComputeDerivedQuantities::run (utils/ComputeDerivedQuantities.h:96-180): the
// derived quantities of a cell's conservative state that `need` asks for, FP64
// in the reference's operation order.  d[q]: 0 RHO_MIX, 1 THERMAL_PRESSURE,
// 2 SPEED_OF_SOUND, 3 SPECIFIC_EKIN, 4 LOCAL_MACH_NUMBER, 5 VX, 6 VY, 7 VZ
// (the DERIVED_QUANTITY enum order).
template <int DIM>
__device__ __forceinline__ void
derived_ref64(const double * u, int need, const PhysParams & P, double * d)
{
  using H = V<DIM>;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    d[k] = 0.0;
  d[0] = u[H::ID];
  if (need & (NEED_PRESSURE | NEED_EKIN))
  {
    // compute_mixture_ekin (models/utils.h:124-151): density from ID
    const double rho = fmax(u[H::ID], P.smallr);
    const double ux = u[H::IU] / rho, uy = u[H::IV] / rho;
    double       ekin;
    if constexpr (DIM == 2)
      ekin = 0.5 * (ux * ux + uy * uy);
    else
    {
      const double uz = u[H::IW] / rho;
      ekin = 0.5 * (ux * ux + uy * uy + uz * uz);
    }
    d[3] = ekin;
    if (need & NEED_PRESSURE)
    {
      // compute_mixture_pressure (models/utils.h:160-185): density from the partial densities
      const double dm = fmax(u[H::IAD0] + u[H::IAD1], P.smallr);
      const double eint = u[H::IE] / dm - ekin;
      const double a0 = u[H::IA0];
      if (!P.mg_any)
        d[1] = (dm * eint - eosPI(P, a0, 1 - a0)) / eosS(P, a0, 1 - a0);
      else
      {
        double S, PI, C1, C0;
        mg_mixture(P, a0, 1 - a0, u[H::IAD0], u[H::IAD1], S, PI, C1, C0);
        d[1] = (dm * eint - PI) / S;
      }
    }
  }
  if (need & (NEED_SOUND | NEED_MACH | NEED_VELOCITY))
  {
    double q[7];
    d[2] = prim_fp64<DIM>(u, q, P);
    d[5] = q[H::QU];
    d[6] = q[H::QV];
    double un = q[H::QU] * q[H::QU] + q[H::QV] * q[H::QV];
    if constexpr (DIM == 3)
    {
      d[7] = q[H::QW];
      un += q[H::QW] * q[H::QW];
    }
    if (need & NEED_MACH)
      d[4] = sqrt(un) / d[2];
  }
}

struct Derived64
{
  double v[8];
};

// one call per cell: with a call per quantity, each converting the cell again,
// eight quantities of 486k cells that all take it were 479 us, of constants
// outside the fast form's range 559 us; 184 and 186 us this way
template <int DIM>
__device__ __noinline__ Derived64
derived_cold64(State64<DIM> s, int need, const PhysParams * P)
{
  Derived64 r;
  derived_ref64<DIM>(s.v, need, *P, r.v);
  return r;
}

// the same from the fast operations; false when a value leaves the range of
// g5_fast64.cuh
template <int DIM, bool MG>
__device__ __forceinline__ bool
derived_fast64(const double * u, int need, const PhysParams & P, double * d)
{
  using H = V<DIM>;
  bool          bad = false;
  const bool    stiff = mixture_stiff64<MG>(P);
  const double  rho = max_pos64(u[H::ID], P.smallr);
  const Recip64 rd = recip64(rho, bad);
  const double  ux = quot64(u[H::IU], rd, bad), uy = quot64(u[H::IV], rd, bad);
  double        k2 = mul64(ux, ux, bad) + mul64(uy, uy, bad);
  bad = bad || x64_raw_bad(rho) || x64_raw_bad(u[H::IU]) || x64_raw_bad(u[H::IV]);
  d[5] = ux;
  d[6] = uy;
  d[7] = 0.0;
  if constexpr (DIM == 3)
  {
    d[7] = quot64(u[H::IW], rd, bad);
    k2 = k2 + mul64(d[7], d[7], bad);
    bad = bad || x64_raw_bad(u[H::IW]);
  }
  d[3] = 0.5 * k2;
  if (need & (NEED_PRESSURE | NEED_SOUND | NEED_MACH))
  {
    const double a0u = u[H::IA0], a1u = 1.0 - a0u;
    Mix64        m = mixture64<MG>(P, a0u, a1u, u[H::IAD0], u[H::IAD1], bad);
    // the mixture pressure takes the density of the partial densities in the
    // internal energy, the primitives' pressure ID: usually the same number
    const double dm = max_pos64(u[H::IAD0] + u[H::IAD1], P.smallr);
    bad = bad || x64_raw_bad(u[H::IE]) || x64_raw_bad(a0u) || x64_raw_bad(u[H::IAD0]) || x64_raw_bad(u[H::IAD1]);
    const bool same = bits64(dm) == bits64(rho);
    double     p = 0.0;
    if ((need & (NEED_SOUND | NEED_MACH)) || same)
    {
      const double n = mul64(rho, __fma_rn(-0.5, k2, quot64(u[H::IE], rd, bad)), bad);
      p = div64(add_if64(stiff, n, neg64(m.PI)), m.S, bad);
    }
    d[1] = p;
    if ((need & NEED_PRESSURE) && !same)
    {
      const double n = mul64(dm, __fma_rn(-0.5, k2, div64(u[H::IE], dm, bad)), bad);
      d[1] = div64(add_if64(stiff, n, neg64(m.PI)), m.S, bad);
    }
    if (need & (NEED_SOUND | NEED_MACH))
    {
      const double a0 = clamp_a64(a0u);
      const double r0 = clamp_r64(u[H::IAD0]), r1 = clamp_r64(u[H::IAD1]);
      if (bits64(a0) != bits64(a0u) || (MG && (bits64(r0) != bits64(u[H::IAD0]) || bits64(r1) != bits64(u[H::IAD1]))))
        m = mixture64<MG>(P, a0, 1.0 - a0, r0, r1, bad);
      d[2] = sound64(rho, p, m, stiff, bad);
      if (need & NEED_MACH)
        d[4] = div64(sqrt64(k2, bad), d[2], bad);
    }
  }
  return !bad;
}

// The fields of one output file (SolverGodunovFiveEq::save_solution_hdf5,
// SolverGodunovFiveEq.cpp:809-886: each a per-quadrant dataset of the state's
// variables or of a derived quantity) for blocks [oct_begin, oct_begin +
// num_octs), in one pass over U: field k of cell g (counted from oct_begin) to
// out[k * stride + g] (FieldList codes: a variable of U, or FIELD_DERIVED + a
// derived quantity).  KIND 0, 1 (stiffened gases, Mie-Grueneisen laws): the
// derived quantities from the fast operations; 2: in the reference's
// arithmetic.  12 fields (4 derived) of 486k cells: 262 us with the reference
// arithmetic per field, 37 us from the fast operations, 164 us in KIND 2.
template <int DIM, int B, int KIND>
__global__ void __launch_bounds__(256)
fields_kernel(const double * __restrict__ U, double * __restrict__ out, const __grid_constant__ FieldList fl, long long stride, long long oct_begin,
              long long num_octs, const __grid_constant__ PhysParams P)
{
  using H = V<DIM>;
  constexpr int   NC = DIM == 2 ? B * B : B * B * B;
  const long long total = num_octs * NC;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long long)gridDim.x * blockDim.x)
  {
    const long long oct = oct_begin + g / NC;
    const int       cell = (int)(g % NC);
    double          u[H::NV], d[8];
#pragma unroll
    for (int v = 0; v < H::NV; ++v)
      u[v] = U[(oct * H::NV + v) * NC + cell];
    d[0] = u[H::ID];
    if (fl.need != 0)
    {
      bool fast = false;
      if constexpr (KIND != 2)
        fast = derived_fast64<DIM, KIND == 1>(u, fl.need, P, d);
      if (!fast)
      {
        State64<DIM> s;
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          s.v[v] = u[v];
        const Derived64 r = derived_cold64<DIM>(s, fl.need, &P);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          d[q] = r.v[q];
      }
      d[0] = u[H::ID];
    }
    for (int k = 0; k < fl.n; ++k)
    {
      const int c = fl.code[k];
      double    r = 0.0;
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
        r = c == v ? u[v] : r;
      if (c >= FIELD_DERIVED)
      {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          r = c == FIELD_DERIVED + q ? d[q] : r;
      }
      out[k * stride + g] = r;
    }
  }
}

} // namespace g5
