// g5_step3d_f64.cuh — the 3D block timestep in FP64 with the fast arithmetic
// of g5_fast64.cuh (MG: the Mie-Grueneisen mixture rules).  The phases, the shared arrays and the
// coarse/fine records are those of step3d_kernel (g5_step3d.cuh), whose FP64
// form is the reference arithmetic; the results are the same doubles.
//
// One CTA of 576 threads per 8^3 block: the 576 faces of a direction take one
// round (512 threads took two, the second with 64 faces), at 96 registers (what
// 18 warps leave each; 388 bytes of spill stores, with the general laws 658).
// The three directions run through one copy of the face code (a run-time
// direction): three would not fit the instruction cache.  A value outside the
// fast form's range sends the rest of the block to the reference arithmetic
// (the `cold` functions).
#pragma once

#include "g5_fast64.cuh"
#include "g5_step3d.cuh"

namespace g5
{

struct Step3D64
{
  using T = Step3DTraits<false>;
  static constexpr int NT = 576;
  static constexpr int NTHINC = 640; // cells with a face of one direction
  // sQ, sHS, the mixture's S of the ring, the face fluxes of one direction,
  // the direction's THINC face values (right, left) and the list of those
  // that have one
  static constexpr int OFF_HS = T::NQ * T::GGG, OFF_S = OFF_HS + T::NHS * T::SSS, OFF_F = OFF_S + T::SSS;
  static constexpr int OFF_AF = OFF_F + T::NF * T::NFF;
  static constexpr size_t smem_bytes = sizeof(double) * (size_t)(OFF_AF + 2 * NTHINC) + 2 * NTHINC + 64;
  static_assert(NT == T::NFF, "one round of faces per direction");
};

// the unit stride of a direction in the ghosted (12^3) and ring (10^3) arrays
__device__ __forceinline__ int
ghost_stride3(int dir)
{
  return dir == 0 ? 1 : (dir == 1 ? Step3D64::T::G : Step3D64::T::GG);
}
__device__ __forceinline__ int
ring_stride3(int dir)
{
  return dir == 0 ? 1 : (dir == 1 ? Step3D64::T::S : Step3D64::T::SS);
}

// Hancock source of one face-neighbour cell (hancock_ref3 in the fast
// operations) and the mixture's S; true when a value left the range
template <bool MG>
__device__ __forceinline__ bool
hancock_fast3(const double * sQ, double * sHS, double * sS, int gi, int r, double dtdx, const PhysParams & P)
{
  using T = Step3D64::T;
  constexpr int G = T::G, GG = T::GG, GGG = T::GGG, SSS = T::SSS;
  bool          bad = false;
  const double  a0 = sQ[6 * GGG + gi], a1 = 1.0 - a0;
  const Mix64   m = mixture64<MG>(P, a0, a1, sQ[gi], sQ[GGG + gi], bad);
  sS[r] = m.S;
  if (P.integrator != 0)
    return bad;
  const int     st = P.st64;
  const bool    stiff = mixture_stiff64<MG>(P);
  const double  p = sQ[2 * GGG + gi];
  const double  rr = sQ[gi] + sQ[GGG + gi];
  const Recip64 rd = recip64(rr, bad);
  const double  c = sound64(rr, p, m, stiff, bad);
  // each source is a sum over the directions, x first
  double sr = 0.0, sp = 0.0, sv[3] = { 0.0, 0.0, 0.0 };
#pragma unroll
  for (int e = 0; e < 3; ++e)
  {
    const int o = e == 0 ? 1 : (e == 1 ? G : GG);
    double    d[6];
#pragma unroll
    for (int k = 0; k < 6; ++k)
    {
      const double * Qk = sQ + k * GGG + gi;
      d[k] = st != 0 ? slope_fast64(Qk[0], Qk[o], Qk[-o], st, bad) : 0.0;
    }
    const double mu = neg64(sQ[(3 + e) * GGG + gi]);
    const double dr = mul64(d[3 + e], rr, bad);
    const double tr = mul64(mulh64(mu, d[0] + d[1], bad) - dr, dtdx, bad);
    const double tp = mul64(mulh64(mu, d[2], bad) - mulh64(mul64(dr, c, bad), c, bad), dtdx, bad);
    sr = e == 0 ? tr : sr + tr;
    sp = e == 0 ? tp : sp + tp;
#pragma unroll
    for (int f = 0; f < 3; ++f)
    {
      double t = mulh64(mu, d[3 + f], bad);
      if (f == e)
        t = t - quot64(d[2], rd, bad);
      t = mul64(t, dtdx, bad);
      sv[f] = e == 0 ? t : sv[f] + t;
    }
  }
  sHS[r] = mul64(sr, a0, bad);
  sHS[SSS + r] = mul64(sr, a1, bad);
  sHS[2 * SSS + r] = sp;
#pragma unroll
  for (int f = 0; f < 3; ++f)
    sHS[(3 + f) * SSS + r] = sv[f];
  return bad;
}

__device__ __noinline__ void
hancock_cold3(const double * sQ, double * sHS, int gi, int r, double dtdx, const PhysParams * P)
{
  hancock_ref3(sQ, sHS, gi, r, dtdx, *P);
}

// the state of one face side beyond its linear reconstruction q: THINC values
// (ti: the cell's entry) or the floor of the partial densities.  Returns the
// mixture's S; gi, si: the cell in the ghosted and ring arrays, af the side's
// THINC values
__device__ __forceinline__ double
face_side_fast3(const double * sQ, const double * sHS, const double * sS, const double * af_side, int gi, int si, int ti, const PhysParams & P, double * q,
                bool & bad)
{
  using T = Step3D64::T;
  constexpr int GGG = T::GGG, SSS = T::SSS;
  const double  a0 = sQ[6 * GGG + gi];
  double        S = sS[si];
  q[6] = a0;
  if (P.thinc)
  {
    const double af = af_side[ti];
    if (bits64(af) != bits64(thinc_none64()))
    {
      const bool        hancock = P.integrator == 0;
      const ThincSide64 t = thinc_side64(a0, af, sQ[gi], sQ[GGG + gi], hancock ? sHS[si] : 0.0, hancock ? sHS[SSS + si] : 0.0, &P);
      q[0] = t.q0;
      q[1] = t.q1;
      q[6] = af;
      S = t.S;
      bad = bad || t.bad;
    }
  }
  else
  {
    q[0] = max_pos64(q[0], P.smallr);
    q[1] = max_pos64(q[1], P.smallr);
  }
  return S;
}

__device__ __noinline__ void
face_flux_cold3(const double * sQ, const double * sHS, double * sF, int f, int dir, double dtdx, const PhysParams * P)
{
  if (dir == 0)
    face_flux3<0>(sQ, sHS, f, sF, dtdx, *P);
  else if (dir == 1)
    face_flux3<1>(sQ, sHS, f, sF, dtdx, *P);
  else
    face_flux3<2>(sQ, sHS, f, sF, dtdx, *P);
}

// the THINC entry of the cell (x, y, z) of direction dir: 10 cells along it,
// 8 x 8 across
__device__ __forceinline__ int
thinc_index3(int dir, int x, int y, int z)
{
  return dir == 0 ? (x + 1) + 10 * (y + 8 * z) : (dir == 1 ? x + 8 * ((y + 1) + 10 * z) : x + 8 * (y + 8 * (z + 1)));
}

// the entry's cell in the ghosted arrays
__device__ __forceinline__ int
thinc_ghost3(int dir, int i)
{
  using T = Step3D64::T;
  const int ex = dir == 0 ? 10 : 8, ey = dir == 1 ? 10 : 8;
  const int x = i % ex - (dir == 0), y = (i / ex) % ey - (dir == 1), z = i / (ex * ey) - (dir == 2);
  return (x + 2) + T::G * (y + 2) + T::GG * (z + 2);
}

// lists the cells of direction dir that take the THINC profile, marks the others
__device__ __forceinline__ void
thinc_list3(const double * sQ, double * sAF, short * sList, int * count, int dir, const PhysParams & P)
{
  const int o = ghost_stride3(dir);
  for (int i = threadIdx.x; i < Step3D64::NTHINC; i += Step3D64::NT)
  {
    const double * A = sQ + 6 * Step3D64::T::GGG + thinc_ghost3(dir, i);
    if (thinc_cell64(A[0], A[-o], A[o], P))
      sList[atomicAdd(count, 1)] = (short)i;
    else
      sAF[i] = sAF[Step3D64::NTHINC + i] = thinc_none64();
  }
}

// an entry's face values on both sides
__device__ __forceinline__ bool
thinc_eval3(const double * sQ, double * sAF, int dir, int i, const PhysParams & P)
{
  using T = Step3D64::T;
  constexpr int  G = T::G, GG = T::GG;
  const double * A = sQ + 6 * T::GGG + thinc_ghost3(dir, i);
  // (1, 2, 1) x (1, 2, 1)-weighted central differences (youngs_abs_3d; the
  // weights are powers of two, so each fused term rounds as the two-step one)
  double g[3] = { 0.0, 0.0, 0.0 };
#pragma unroll 1
  for (int c = -1; c <= 1; ++c)
#pragma unroll 1
    for (int b = -1; b <= 1; ++b)
    {
      const double w = (b == 0 ? 2.0 : 1.0) * (c == 0 ? 2.0 : 1.0);
      g[0] = __fma_rn(w, A[1 + G * b + GG * c] - A[-1 + G * b + GG * c], g[0]);
      g[1] = __fma_rn(w, A[b + G + GG * c] - A[b - G + GG * c], g[1]);
      g[2] = __fma_rn(w, A[b + G * c + GG] - A[b + G * c - GG], g[2]);
    }
  bool         bad = false;
  const double n2 = (g[0] * g[0] + g[1] * g[1]) + g[2] * g[2];
  const double nd = youngs_ratio64(dir == 0 ? g[0] : (dir == 1 ? g[1] : g[2]), n2, bad);
  const int    o = ghost_stride3(dir);
  thinc_pair64(A[0], A[-o], A[o], nd, P, sAF[i], sAF[Step3D64::NTHINC + i], bad);
  return bad;
}

// HLLC flux of face f of direction dir, scaled by dt/dx (face_flux3)
template <bool MG>
__device__ __forceinline__ bool
face_flux_fast3(const double * sQ, const double * sHS, const double * sS, const double * sAF, double * sF, int f, int dir, double dtdx, const PhysParams & P)
{
  using T = Step3D64::T;
  using H = V<3>;
  constexpr int B = T::B, G = T::G, GG = T::GG, GGG = T::GGG, S = T::S, SS = T::SS, SSS = T::SSS, NFF = T::NFF;
  const int     ex = B + (dir == 0), ey = B + (dir == 1);
  const int     fi = f % ex, fj = (f / ex) % ey, fk = f / (ex * ey);
  const int     gR = (fi + 2) + G * (fj + 2) + GG * (fk + 2), sR = (fi + 1) + S * (fj + 1) + SS * (fk + 1);
  const int     o = ghost_stride3(dir);
  double        qL[7], qR[7], fl[9];
  bool          bad = false;
  // both sides' linear states (face_state3, the normal velocity first):
  // of a component's four values across the face, the middle difference serves
  // both slopes
  const int     sL = sR - ring_stride3(dir), st = P.st64;
  const bool    hancock = P.integrator == 0;
#pragma unroll
  for (int k = 0; k < 6; ++k)
  {
    const int      from = k < 3 ? k : (k == 3 ? 3 + dir : (k == 3 + dir ? 3 : k));
    const double * Q = sQ + from * GGG + gR;
    const double   b = Q[-o], c = Q[0];
    qL[k] = b;
    qR[k] = c;
    if (st != 0)
    {
      const double a_ = Q[-2 * o], d = Q[o], m = c - b;
      qL[k] = __fma_rn(0.5, limit_fast64(b - a_, m, c, a_, st, bad), b);
      qR[k] = __fma_rn(-0.5, limit_fast64(m, d - c, d, b, st, bad), c);
    }
    if (hancock)
    {
      qL[k] = __fma_rn(0.5, sHS[from * SSS + sL], qL[k]);
      qR[k] = __fma_rn(0.5, sHS[from * SSS + sR], qR[k]);
    }
  }
  const double  Sl = face_side_fast3(sQ, sHS, sS, sAF, gR - o, sL, thinc_index3(dir, fi - (dir == 0), fj - (dir == 1), fk - (dir == 2)), P, qL, bad);
  const double  Sr = face_side_fast3(sQ, sHS, sS, sAF + Step3D64::NTHINC, gR, sR, thinc_index3(dir, fi, fj, fk), P, qR, bad);
  const Side64  L = hllc_side64<3, MG>(qL, Sl, P, bad);
  const Side64  R = hllc_side64<3, MG>(qR, Sr, P, bad);
  hllc_fast64<3>(qL, qR, L, R, dtdx, fl, bad);
  if (bad)
  {
    face_flux_cold3(sQ, sHS, sF, f, dir, dtdx, &P);
    return true;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k)
    sF[(k == H::FU ? H::FU + dir : (k >= H::FV && k == H::FU + dir ? H::FU : k)) * NFF + f] = fl[k];
  return false;
}

// end of the update of a cell whose values left the range: the reference's
// renormalisation and CFL rate; writes the cell (variables NC apart)
__device__ __noinline__ double
finish_cold3(State64<3> s, double * out, double dx, const PhysParams * P, bool want_dt)
{
  using H = V<3>;
  double *     u2 = s.v;
  const double inv = 1.0 / (u2[H::IA0] + u2[H::IA1]);
  u2[H::ID] = u2[H::IAD0] + u2[H::IAD1];
  u2[H::IA0] *= inv;
  u2[H::IA1] *= inv;
  for (int v = 0; v < H::NV; ++v)
    out[v * 512] = u2[v];
  if (!want_dt)
    return 0.0;
  double       q[7];
  const double c = prim_fp64<3>(u2, q, *P);
  return (c + fabs(q[H::QU])) / dx + (c + fabs(q[H::QV])) / dx + (c + fabs(q[H::QW])) / dx;
}

__device__ __noinline__ double2
source_cold3(State64<3> s, const PhysParams * P)
{
  double2 st;
  source_factors_fp64<3>(s.v, *P, st.x, st.y);
  return st;
}

__device__ __forceinline__ State64<3>
pack_state3(const double * u)
{
  State64<3> s;
#pragma unroll
  for (int v = 0; v < V<3>::NV; ++v)
    s.v[v] = u[v];
  return s;
}

template <bool MG>
__global__ void __launch_bounds__(Step3D64::NT, 1)
step3d_fast64_kernel(const __grid_constant__ StepArgs a)
{
  using T = Step3D64::T;
  using H = V<3>;
  constexpr int B = T::B, NT = Step3D64::NT, G = T::G, GG = T::GG, GGG = T::GGG, S = T::S, SS = T::SS, NC = 512;
  constexpr int NFF = T::NFF;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *           sQ = reinterpret_cast<double *>(smem_raw);
  double *           sHS = sQ + Step3D64::OFF_HS;
  double *           sS = sQ + Step3D64::OFF_S;
  double *           sF = sQ + Step3D64::OFF_F;
  double *           sAF = sQ + Step3D64::OFF_AF;
  short *            sList = reinterpret_cast<short *>(sAF + 2 * Step3D64::NTHINC);
  __shared__ int     sThinc[2]; // entries of the list of the current and the next direction
  __shared__ double  sRed[NT / 32];
  __shared__ int     sSlot[12]; // the block's reflux slots (faces 0-5), then its defer slots
  __shared__ int     sNext;     // the CTA's next block
  const int          tid = threadIdx.x;
  const PhysParams & P = a.p;
  const bool         owner = tid < NC;
  const int          ci = tid % B, cj = (tid / B) % B, ck = tid / (B * B);

  const int nwalk = step_count(a);
  if (tid < 2)
    sThinc[tid] = 0;
  for (int iw = blockIdx.x; iw < nwalk;)
  {
    const int    n = a.work ? a.work[iw] : iw;
    // the next block is claimed now (the ticket's latency hides behind the gather)
    const int    next_v = tid == 12 ? claim_next(a, iw, nwalk) : 0;
    const int    ins = a.m.inst ? a.m.inst[n] : 0;
    const double dx = P.level_dx[a.m.level[n]];
    const int    c0[3] = { a.m.coord[n * 3 + 0], a.m.coord[n * 3 + 1], a.m.coord[n * 3 + 2] };
    int          slot_v = -1; // coarse/fine slots, stored to shared memory after the gather
    if (a.m.reflux_slot && tid < 12)
      slot_v = tid < 6 ? a.m.reflux_slot[n * 6 + tid] : a.m.defer_slot[n * 6 + tid - 6];
    // a value left the fast form's range (per thread until the next barrier,
    // then for the CTA)
    double dtdx = a.dt[ins];
    bool   cold = x64_raw_bad(dtdx) || x64_raw_bad(dx);
    {
      const double q = div64(dtdx, dx, cold);
      dtdx = cold ? div_cold64(dtdx, dx) : q;
    }

    // ---------------- phase 1: own cell + halo -> primitives (the threads
    // without a cell take the first halo cells)
    const double * own = a.U + (size_t)n * H::NV * NC + tid;
    const int      nhalo = HALO3_FULL + (P.thinc != 0 ? HALO3_ALPHA : 0);
    // the own cell is the walk's first item of the threads that have one
    for (int it = owner ? -1 : 0, h = owner ? 0 : tid - NC; it < 0 || h < nhalo; ++it)
    {
      int    gidx;
      double u[H::NV];
      if (it < 0)
      {
        gidx = (ci + 2) + G * (cj + 2) + GG * (ck + 2);
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          u[v] = own[v * NC];
        h = tid + NT - NC;
      }
      else
      {
        int g[3];
        halo_coords_3d(h, g);
        gidx = (g[0] + 2) + G * (g[1] + 2) + GG * (g[2] + 2);
        if (h >= HALO3_FULL)
        {
          if (!gather_ghost_3d<true>(a, n, c0, g, u))
          {
            raise_status(a.status, STATUS_MESH);
            u[H::IA0] = a.U[((size_t)n * H::NV + H::IA0) * NC + tid % NC];
          }
          const bool b = x64_raw_bad(u[H::IA0]);
          cold = cold || b;
          sQ[6 * GGG + gidx] = b ? alpha_prim<false>(u[H::IA0]) : clamp_a64(u[H::IA0]);
          h += NT;
          continue;
        }
        if (!gather_ghost_3d(a, n, c0, g, u))
        {
          raise_status(a.status, STATUS_MESH);
          const double * cell = a.U + (size_t)n * H::NV * NC + tid % NC;
#pragma unroll
          for (int v = 0; v < H::NV; ++v)
            u[v] = cell[v * NC];
        }
        h += NT;
      }
      double q[7];
      bool   bad = false;
      prim_fast64<3, false, true, MG>(u, q, P, bad);
      if (bad)
      {
        cold = true;
        prim_ref64<3>(pack_state3(u), &P, sQ + gidx, GGG);
      }
      else
      {
#pragma unroll
        for (int k = 0; k < 7; ++k)
          sQ[k * GGG + gidx] = q[k];
      }
    }
    if (tid < 12)
      sSlot[tid] = slot_v;
    if (tid == 12)
      sNext = next_v;
    cold = __syncthreads_or(cold) != 0;
    // the next block of this CTA: its own cells and table rows into L2
    if (tid < 3 && sNext < nwalk)
    {
      const int nn = a.work ? a.work[sNext] : sNext;
      if (tid == 0)
        prefetch_l2_range(a.U + (size_t)nn * H::NV * NC, (unsigned)(H::NV * NC * sizeof(double)));
      else if (tid == 1)
        prefetch_l2_range(a.m.nbr + (size_t)nn * 27 * 8, 27 * 8 * sizeof(int32_t));
      else
        prefetch_l2_line(a.m.nbr_rel + (size_t)nn * 27);
    }

    // ---------------- phase 2: Hancock source of the 896 face-neighbour cells
    // (the enumeration of step3d_kernel)
    const bool cold0 = cold;
    for (int h = tid; h < NC + 6 * B * B; h += NT)
    {
      int ri, rj, rk;
      if (h < NC)
      {
        ri = h & 7;
        rj = (h >> 3) & 7;
        rk = h >> 6;
      }
      else
      {
        const int i = h - NC, f = i >> 6, pa = i & 7, pb = (i >> 3) & 7;
        const int side = (f & 1) ? B : -1;
        ri = f < 2 ? side : pa;
        rj = f < 2 ? pa : (f < 4 ? side : pb);
        rk = f < 4 ? pb : side;
      }
      const int r = (ri + 1) + S * (rj + 1) + SS * (rk + 1);
      const int gi = (ri + 2) + G * (rj + 2) + GG * (rk + 2);
      bool      bad = cold0;
      if (!bad)
        bad = hancock_fast3<MG>(sQ, sHS, sS, gi, r, dtdx, P);
      if (bad)
      {
        cold = true;
        hancock_cold3(sQ, sHS, gi, r, dtdx, &P);
      }
    }

    // the owned cell: its running state (read again, an L2 hit), and the
    // volume-fraction source factors
    double u2[H::NV], st0 = 1.0, st1 = 1.0;
    double a0n = 0.0, a1n = 0.0;
    if (owner)
    {
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
        u2[v] = __ldcg(own + v * NC);
      a0n = u2[H::IA0];
      a1n = u2[H::IA1];
      if (P.source_term == 1)
      {
        bool bad = cold0;
        if (!bad)
          source_factors_fast64<3, MG>(u2, P, st0, st1, bad);
        if (bad)
        {
          const double2 st = source_cold3(pack_state3(u2), &P);
          st0 = st.x;
          st1 = st.y;
        }
      }
      cold = cold || x64_raw_bad(a1n) || x64_raw_bad(st0) || x64_raw_bad(st1);
    }
    if (P.thinc != 0)
      thinc_list3(sQ, sAF, sList, &sThinc[0], 0, P);
    cold = __syncthreads_or(cold) != 0;

    // deferred cells (next to a finer face) are finished by reflux3d_kernel
    const int * dsl = a.m.defer_slot ? sSlot + 6 : nullptr;
    bool        deferred = false;
    if (dsl && owner)
    {
      const int cc[3] = { ci, cj, ck };
#pragma unroll
      for (int f = 0; f < 6; ++f)
        deferred = deferred || (dsl[f] >= 0 && cc[f >> 1] == ((f & 1) ? B - 1 : 0));
    }

#pragma unroll 1
    for (int dir = 0; dir < 3; ++dir)
    {
      // ---------------- phase 3: one face per thread, after the direction's
      // THINC values (listed before the last barrier)
      if (P.thinc != 0 && sThinc[dir & 1] > 0 && !cold)
      {
        for (int i = tid; i < sThinc[dir & 1]; i += NT)
          cold |= thinc_eval3(sQ, sAF, dir, sList[i], P);
        cold = __syncthreads_or(cold) != 0;
      }
      bool bad = cold;
      if (!bad)
        bad = face_flux_fast3<MG>(sQ, sHS, sS, sAF, sF, tid, dir, dtdx, P);
      else
        face_flux_cold3(sQ, sHS, sF, tid, dir, dtdx, &P);
      cold = __syncthreads_or(bad) != 0;
      if (tid == 0)
        sThinc[dir & 1] = 0;
      if (P.thinc != 0 && dir < 2)
        thinc_list3(sQ, sAF, sList, &sThinc[(dir + 1) & 1], dir + 1, P);

      // face index of the owned cell's left/right face in this direction
      const int ext0 = B + (dir == 0), ext1 = B + (dir == 1);
      const int il = ci + ext0 * (cj + ext1 * ck);
      const int ir = il + (dir == 0 ? 1 : (dir == 1 ? ext0 : ext0 * ext1));

      // ---------------- publish coarse/fine records of this direction (AMR only)
      if (a.m.reflux_slot)
      {
        for (int side = 0; side < 2; ++side)
        {
          const int rs = sSlot[2 * dir + side];
          // positions along the face: the two transverse coordinates (first, second)
          if (rs >= 0 && tid < B * B)
          {
            const int t1 = tid % B, t2 = tid / B, edge = side ? B : 0;
            const int fx = dir == 0 ? edge : t1, fy = dir == 1 ? edge : (dir == 0 ? t1 : t2), fz = dir == 2 ? edge : t2;
            const int fidx = fx + ext0 * (fy + ext1 * fz);
            double *  dst = a.reflux_buf + ((size_t)rs * B * B + tid) * 9;
#pragma unroll
            for (int k = 0; k < 9; ++k)
              dst[k] = sF[k * NFF + fidx];
          }
        }
        // own face fluxes of deferred cells, this direction (left then right)
        if (deferred)
        {
          for (int f = 0; f < 6; ++f)
          {
            const int d2 = f >> 1;
            if (dsl[f] < 0 || (d2 == 0 ? ci : (d2 == 1 ? cj : ck)) != ((f & 1) ? B - 1 : 0))
              continue;
            const int t1 = d2 == 0 ? cj : ci, t2 = d2 == 2 ? cj : ck;
            double *  dst = a.defer_buf + (((size_t)dsl[f] * B * B + t1 + B * t2) * 6 + 2 * dir) * 9;
#pragma unroll
            for (int k = 0; k < 9; ++k)
            {
              dst[k] = sF[k * NFF + il];
              dst[9 + k] = sF[k * NFF + ir];
            }
          }
        }
      }

      // ---------------- phase 4: this direction's update of the owned cell
      // (the reference starts each sum from 0 + F_left: the same value but
      // for the sign of a zero)
      if (owner && !deferred)
      {
        const double usl = sF[H::FUS * NFF + il], usr = sF[H::FUS * NFF + ir];
        if (cold)
        {
          double acc[8];
#pragma unroll
          for (int k = 0; k < 8; ++k)
            acc[k] = 0.0 + sF[k * NFF + il];
          acc[H::FA0] -= st0 * usl * a0n;
          acc[H::FA1] -= st1 * usl * a1n;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            acc[k] = acc[k] - sF[k * NFF + ir];
          acc[H::FA0] += st0 * usr * a0n;
          acc[H::FA1] += st1 * usr * a1n;
          apply_dir_fp64(u2, acc);
        }
        else
        {
          const bool mp = P.source_term == 1;
          bool       b2 = false;
          double     i0 = alpha_inc64(sF[H::FA0 * NFF + il], sF[H::FA0 * NFF + ir], usl, usr, st0, a0n, mp, b2);
          double     i1 = alpha_inc64(sF[H::FA1 * NFF + il], sF[H::FA1 * NFF + ir], usl, usr, st1, a1n, mp, b2);
          if (b2)
          {
            i0 = (sF[H::FA0 * NFF + il] - st0 * usl * a0n) - sF[H::FA0 * NFF + ir] + st0 * usr * a0n;
            i1 = (sF[H::FA1 * NFF + il] - st1 * usl * a1n) - sF[H::FA1 * NFF + ir] + st1 * usr * a1n;
          }
          u2[H::IAD0] = clamp_r64(u2[H::IAD0] + (sF[H::FR0 * NFF + il] - sF[H::FR0 * NFF + ir]));
          u2[H::IAD1] = clamp_r64(u2[H::IAD1] + (sF[H::FR1 * NFF + il] - sF[H::FR1 * NFF + ir]));
          u2[H::IA0] = clamp_a64(u2[H::IA0] + i0);
          u2[H::IA1] = clamp_a64(u2[H::IA1] + i1);
          u2[H::IE] += sF[H::FE * NFF + il] - sF[H::FE * NFF + ir];
          u2[H::IU] += sF[H::FU * NFF + il] - sF[H::FU * NFF + ir];
          u2[H::IV] += sF[H::FV * NFF + il] - sF[H::FV * NFF + ir];
          u2[H::IW] += sF[H::FW * NFF + il] - sF[H::FW * NFF + ir];
        }
      }
      __syncthreads();
    }

    double m_inv = 0.0;
    if (owner && !deferred)
    {
      double * out = a.U2 + (size_t)n * H::NV * NC + tid;
      bool     bad = cold;
      // the state before the renormalisation, for the cold path
      if (!bad)
      {
        const double b0 = u2[H::IA0], b1 = u2[H::IA1];
        m_inv = finish_fast64<3, MG>(u2, dx, P, a.invdt != nullptr, bad);
        if (bad)
        {
          u2[H::IA0] = b0;
          u2[H::IA1] = b1;
        }
      }
      if (bad)
      {
        m_inv = finish_cold3(pack_state3(u2), out, dx, &P, a.invdt != nullptr);
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          u2[v] = out[v * NC];
      }
      bool finite = true;
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
      {
        out[v * NC] = u2[v];
        finite = finite && finite_bits(u2[v]);
      }
      if (!finite)
        raise_status(a.status, STATUS_NONPHYSICAL);
    }
    if (a.invdt)
    {
      m_inv = warp_max_pos64(m_inv);
      if ((tid & 31) == 0)
        sRed[tid >> 5] = m_inv;
      __syncthreads();
      if (tid == 0)
      {
        double mm = 0.0;
        for (int w = 0; w < NT / 32; ++w)
          mm = bits64(sRed[w]) > bits64(mm) ? sRed[w] : mm;
        atomic_max_pos(a.invdt + ins, mm);
      }
    }
    const int next = sNext; // read before the barrier: the next block's claim overwrites it
    __syncthreads();
    iw = next;
  }
}

} // namespace g5
