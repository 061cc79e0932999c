// g5_step2d_f64.cuh — the 2D block timestep in FP64 with the fast arithmetic of
// g5_fast64.cuh (MG: the Mie-Grueneisen mixture rules).  The phases, the
// shared arrays and the coarse/fine records are those of step2d_kernel
// (g5_step2d.cuh), whose FP64 form is the reference arithmetic; the results are
// the same doubles.
//
// A CTA works on a tile of rows [y0, y0 + ty) of a block: a whole block, or in
// 16x16 blocks half or a quarter of one.  Halves cost 10 % more work (the halo
// rows between them), but a launch whose last round of blocks fills at most
// half of the resident CTAs takes that round in halves, one per CTA: 512x32
// shock tube (64 blocks on 152 SMs) 45 -> 31 us per step, 486k-cell AMR
// shock-bubble (6.25 rounds) 388 -> 383 us.
// A value outside the fast form's range sends the cells and faces that read
// it, and the update of the tile, to the reference arithmetic (the `cold`
// functions).  Blocks that hold such values throughout take longer than in
// step2d_kernel (all momenta below 1e-136, 486k cells: 1,397 us against 1,174).
#pragma once

#include "g5_fast64.cuh"
#include "g5_step2d.cuh"

namespace g5
{

template <int B>
struct Step2D64
{
  using T = Step2DTraits<B, false>;
  // more threads than cells, so that the 320 (96) slope cells take one round
  // and the 544 (144) faces two, at 96 (80) registers (16x16: 420 us per
  // shock-bubble step of 486k cells against 444 us with 256 threads at 128
  // registers, 438 us with 384 at 80; 8x8: 147 us against 161 with 64 threads)
  static constexpr int NT = B == 16 ? 320 : 96;
  static constexpr int CTAS = B == 16 ? 2 : 7;
  static constexpr int NREC = 16; // dqx[5] dqy[5] hS[5] and the mixture's S of the cell
  // THINC face values of the 2 B (B + 2) cells and directions, right and
  // left, and the list of those that have one (only with THINC)
  static constexpr int    NTH = 2 * B * (B + 2);
  static constexpr size_t smem_bytes = sizeof(double) * (size_t)(T::NQ * T::G * T::G + NREC * T::S * T::S + 2 * 8 * T::NFF) + 64;
  static constexpr size_t smem_thinc = (2 * sizeof(double) + sizeof(short)) * (size_t)NTH;
  static constexpr bool   SPLIT = B == 16;
};

template <int B>
__device__ __noinline__ void
face_flux_cold64(const double * sQ, const double * sRec, double * sF, int dir, int ff, double dtdx, const PhysParams * P)
{
  face_flux_ref64<B>(sQ, sRec, sF, dir, ff, dtdx, *P);
}

template <int B>
__device__ __noinline__ void
hancock_cold64(const double * sQ, double * sRec, int gi, int r, double dtdx, const PhysParams * P)
{
  hancock_ref64<B>(sQ, sRec, gi, r, dtdx, *P);
}

// the THINC entry (cell, direction) of a tile of ty rows in the arrays sAF:
// (B + 2) ty cells along x, then B (ty + 2) along y
template <int B>
__device__ __forceinline__ int
thinc_index(int dir, int ci, int cj, int ty)
{
  return dir == 0 ? (ci + 1) + (B + 2) * cj : (B + 2) * ty + ci + B * (cj + 1);
}

// the entry's direction and cell
template <int B>
__device__ __forceinline__ void
thinc_cell(int i, int ty, int & dir, int & ci, int & cj)
{
  dir = i < (B + 2) * ty ? 0 : 1;
  const int k = i - dir * (B + 2) * ty;
  ci = dir == 0 ? k % (B + 2) - 1 : k % B;
  cj = dir == 0 ? k / (B + 2) : k / B - 1;
}

// the pair's face values, from its entry
template <int B>
__device__ __forceinline__ bool
thinc_eval2(const double * sQ, double * sRec, double * sAF, int i, int ty, const PhysParams & P)
{
  using T = Step2DTraits<B, false>;
  constexpr int  G = T::G, GG = G * G;
  int            dir, ci, cj;
  thinc_cell<B>(i, ty, dir, ci, cj);
  const double * A = sQ + 5 * GG + (ci + 2) + G * (cj + 2);
  // (1, 2, 1)-weighted central differences (youngs_abs_2d)
  const double gx = (__fma_rn(2.0, A[1], A[1 - G]) + A[1 + G]) - (__fma_rn(2.0, A[-1], A[-1 - G]) + A[-1 + G]);
  const double gy = (__fma_rn(2.0, A[G], A[G - 1]) + A[G + 1]) - (__fma_rn(2.0, A[-G], A[-G - 1]) + A[-G + 1]);
  bool         bad = false;
  const double nd = youngs_ratio64(dir == 0 ? gx : gy, gx * gx + gy * gy, bad);
  const int    o = dir == 0 ? 1 : G;
  thinc_pair64(A[0], A[-o], A[o], nd, P, sAF[i], sAF[Step2D64<B>::NTH + i], bad);
  if (bad) // its faces take the reference arithmetic
    sRec[15 * T::S * T::S + (ci + 1) + T::S * (cj + 1)] = bad_cell64();
  return bad;
}

// FP64: the reconstructed state and the mixture's S of one side (the values
// of face_state_ref64, normal velocity first).  The direction is a run-time
// value: X and Y faces share one copy of the flux code, which is long enough
// to miss the instruction cache.
template <int B>
__device__ __forceinline__ double
face_state_fast64(const double * sQ, const double * sRec, const double * sAF, int ci, int cj, int ty, int dir, int side, const PhysParams & P, double * q,
                  bool & bad)
{
  using T = Step2DTraits<B, false>;
  constexpr int    G = T::G, S = T::S, GG = G * G, SS = S * S;
  const double     off = side > 0 ? 0.5 : -0.5;
  const int        gi = (ci + 2) + G * (cj + 2);
  const int        si = (ci + 1) + S * (cj + 1);
  const double *   dq = sRec + dir * 5 * SS + si;
  const bool       hancock = P.integrator == 0;
#pragma unroll
  for (int k = 0; k < 5; ++k)
  {
    const int    from = k < 3 ? k : (k == 3 ? 3 + dir : 4 - dir);
    const double t = __fma_rn(off, dq[from * SS], sQ[from * GG + gi]);
    q[k] = hancock ? __fma_rn(0.5, sRec[(10 + from) * SS + si], t) : t;
  }
  const double a0 = sQ[5 * GG + gi];
  double       Sm = sRec[15 * SS + si];
  q[5] = a0;
  if (P.thinc)
  {
    const double af = sAF[(side > 0 ? 0 : Step2D64<B>::NTH) + thinc_index<B>(dir, ci, cj, ty)];
    if (bits64(af) != bits64(thinc_none64()))
    {
      const ThincSide64 t = thinc_side64(a0, af, sQ[gi], sQ[GG + gi], hancock ? sRec[10 * SS + si] : 0.0, hancock ? sRec[11 * SS + si] : 0.0, &P);
      q[0] = t.q0;
      q[1] = t.q1;
      q[5] = af;
      Sm = t.S;
      bad = bad || t.bad;
    }
  }
  else
  {
    q[0] = max_pos64(q[0], P.smallr);
    q[1] = max_pos64(q[1], P.smallr);
  }
  return Sm;
}

template <int B, bool MG>
__device__ __forceinline__ bool
face_flux_fast64(const double * sQ, const double * sRec, const double * sAF, double * sF, int ty, int dir, int ff, bool check, double dtdx,
                 const PhysParams & P)
{
  using H = V<2>;
  constexpr int NFF = B * (B + 1), S = B + 2, SS = S * S;
  int           li, lj, ri, rj;
  face_cells<B>(dir, ff, li, lj, ri, rj);
  if (check && (bits64(sRec[15 * SS + (li + 1) + S * (lj + 1)]) == bits64(bad_cell64()) || bits64(sRec[15 * SS + (ri + 1) + S * (rj + 1)]) == bits64(bad_cell64())))
    return true;
  double       qL[6], qR[6], fl[8];
  bool         bad = false;
  const double Sl = face_state_fast64<B>(sQ, sRec, sAF, li, lj, ty, dir, 1, P, qL, bad);
  const double Sr = face_state_fast64<B>(sQ, sRec, sAF, ri, rj, ty, dir, -1, P, qR, bad);
  const Side64 L = hllc_side64<2, MG>(qL, Sl, P, bad);
  const Side64 R = hllc_side64<2, MG>(qR, Sr, P, bad);
  hllc_fast64<2>(qL, qR, L, R, dtdx, fl, bad);
  if (bad)
    return true;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    sF[(k == H::FU ? H::FU + dir : k == H::FV ? H::FV - dir : k) * NFF + ff] = fl[k];
  return false;
}

// the same values (hancock_ref64's) from the fast operations, and the mixture's S of the cell
template <int B, bool MG>
__device__ __forceinline__ bool
hancock_fast64(const double * sQ, double * sRec, int gi, int r, double dtdx, const PhysParams & P)
{
  using T = Step2DTraits<B, false>;
  constexpr int G = T::G, S = T::S, GG = G * G, SS = S * S;
  const bool    stiff = mixture_stiff64<MG>(P), hancock = P.integrator == 0;
  const int     st = P.st64;
  bool          bad = false;
  const double  a0 = sQ[5 * GG + gi], a1 = 1.0 - a0;
  const Mix64   m = mixture64<MG>(P, a0, a1, sQ[gi], sQ[GG + gi], bad);
  sRec[15 * SS + r] = m.S;
  const double rr = sQ[gi] + sQ[GG + gi];
  Recip64      rd = {};
  double       c = 0.0;
  if (hancock)
  {
    rd = recip64(rr, bad);
    c = sound64(rr, sQ[2 * GG + gi], m, stiff, bad);
  }
  // each source is a sum over the two directions, x first; the sums of the
  // normal and transverse velocity change places between them.  (Rolled, as
  // the update's directions are: the instruction cache gains more than the
  // loop costs, 471 -> 461 us with THINC, 386 us without either way.)
  double sr = 0.0, sp = 0.0, sv[2] = { 0.0, 0.0 };
#pragma unroll 1
  for (int e = 0; e < 2; ++e)
  {
    const int o = e == 0 ? 1 : G;
    double    d[5]; // r0 r1 p, normal and transverse velocity
#pragma unroll
    for (int k = 0; k < 5; ++k)
    {
      const int      from = k < 3 ? k : (k == 3 ? 3 + e : 4 - e);
      const double * Qk = sQ + from * GG + gi;
      d[k] = st != 0 ? slope_fast64(Qk[0], Qk[o], Qk[-o], st, bad) : 0.0;
      sRec[(5 * e + from) * SS + r] = d[k];
    }
    if (hancock)
    {
      const double mu = neg64(sQ[(3 + e) * GG + gi]);
      const double dr = mul64(d[3], rr, bad);
      const double tr = mul64(mulh64(mu, d[0] + d[1], bad) - dr, dtdx, bad);
      const double tp = mul64(mulh64(mu, d[2], bad) - mulh64(mul64(dr, c, bad), c, bad), dtdx, bad);
      const double tn = mul64(mulh64(mu, d[3], bad) - quot64(d[2], rd, bad), dtdx, bad);
      const double tt = mul64(mulh64(mu, d[4], bad), dtdx, bad);
      if (e == 0)
      {
        sr = tr;
        sp = tp;
        sv[0] = tn;
        sv[1] = tt;
      }
      else
      {
        sr = sr + tr;
        sp = sp + tp;
        sv[0] = sv[0] + tt;
        sv[1] = sv[1] + tn;
      }
    }
  }
  if (hancock)
  {
    sRec[10 * SS + r] = mul64(sr, a0, bad);
    sRec[11 * SS + r] = mulh64(sr, a1, bad);
    sRec[12 * SS + r] = sp;
    sRec[13 * SS + r] = sv[0];
    sRec[14 * SS + r] = sv[1];
  }
  return bad;
}

// FP64 cold path: the update of a cell whose values leave the fast form's
// range, written to U2 (out, variables NC apart)
template <int B>
__device__ __noinline__ double
update_cold64(State64<2> uin, double * out, const double * sFx, const double * sFy, int ci, int cj, double dx, const PhysParams * P, bool want_dt)
{
  double       u2[V<2>::NV];
  const double r = update_fp64<B>(uin.v, u2, sFx, sFy, ci, cj, dx, *P, want_dt);
  for (int v = 0; v < V<2>::NV; ++v)
    out[v * B * B] = u2[v];
  return r;
}

// update_fp64 from the fast operations.  (The reference
// starts each sum from 0 + F_left: the same value but for the sign of a zero.)
template <int B, bool MG>
__device__ __forceinline__ double
update_fast64(const double * uin, double * u2, const double * sFx, const double * sFy, int ci, int cj, double dx, const PhysParams & P, bool want_dt,
              bool & bad)
{
  using H = V<2>;
  constexpr int NFF = B * (B + 1);
#pragma unroll
  for (int v = 0; v < H::NV; ++v)
    u2[v] = uin[v];
  double     st0, st1;
  const bool mp = P.source_term == 1;
  source_factors_fast64<2, MG>(uin, P, st0, st1, bad);
  bad = bad || x64_raw_bad(uin[H::IA1]); // (the rest was tested for the primitives)
#pragma unroll 1
  for (int dir = 0; dir < 2; ++dir)
  {
    const double * F = dir == 0 ? sFx : sFy;
    const int      il = dir == 0 ? ci + (B + 1) * cj : ci + B * cj;
    const int      ir = dir == 0 ? il + 1 : il + B;
    const double   usl = F[H::FUS * NFF + il], usr = F[H::FUS * NFF + ir];
    u2[H::IAD0] = clamp_r64(u2[H::IAD0] + (F[H::FR0 * NFF + il] - F[H::FR0 * NFF + ir]));
    u2[H::IAD1] = clamp_r64(u2[H::IAD1] + (F[H::FR1 * NFF + il] - F[H::FR1 * NFF + ir]));
    u2[H::IA0] = clamp_a64(u2[H::IA0] + alpha_inc64(F[H::FA0 * NFF + il], F[H::FA0 * NFF + ir], usl, usr, st0, uin[H::IA0], mp, bad));
    u2[H::IA1] = clamp_a64(u2[H::IA1] + alpha_inc64(F[H::FA1 * NFF + il], F[H::FA1 * NFF + ir], usl, usr, st1, uin[H::IA1], mp, bad));
    u2[H::IE] += F[H::FE * NFF + il] - F[H::FE * NFF + ir];
    u2[H::IU] += F[H::FU * NFF + il] - F[H::FU * NFF + ir];
    u2[H::IV] += F[H::FV * NFF + il] - F[H::FV * NFF + ir];
  }
  return finish_fast64<2, MG>(u2, dx, P, want_dt, bad);
}

// halo cell h of a tile of ty rows (4 (B + 4) + 4 ty of them) -> coordinates
// in the tile
template <int B>
__device__ __forceinline__ void
halo_coords_tile(int h, int ty, int & gx, int & gy)
{
  constexpr int G = B + 4;
  if (h < 4 * G)
  {
    const int row = h / G;
    gx = h % G - 2;
    gy = row < 2 ? row - 2 : ty + row - 2;
    return;
  }
  const int c = (h - 4 * G) & 3;
  gy = (h - 4 * G) >> 2;
  gx = c < 2 ? c - 2 : B + c - 2;
}

// n_full: whole blocks at the head of the walk; the n_items - n_full items
// after them are the 2^split tiles each of the blocks that follow (n_full =
// n_items: none)
template <int B, bool MG>
__global__ void __launch_bounds__(Step2D64<B>::NT, Step2D64<B>::CTAS)
step2d_fast64_kernel(const __grid_constant__ StepArgs a, int n_full, int n_items, int split)
{
  using K = Step2D64<B>;
  using T = typename K::T;
  using H = V<2>;
  constexpr int NT = K::NT, G = T::G, S = T::S, GG = T::G * T::G, SS = T::S * T::S, NC = B * B, NFF = T::NFF;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *           sQ = reinterpret_cast<double *>(smem_raw);
  double *           sRec = sQ + T::NQ * GG;
  double *           sFx = sRec + K::NREC * SS; // [8][NFF]  X faces (B+1) x ty
  double *           sFy = sFx + 8 * NFF;       // [8][NFF]  Y faces B x (ty+1)
  double *           sAF = sFy + 8 * NFF;       // THINC face values, then the list
  short *            sList = reinterpret_cast<short *>(sAF + 2 * K::NTH);
  __shared__ double  sRed[NT / 32];
  __shared__ int     sSlot[10]; // the block's reflux slots (faces 0-3), its defer slots, its outside-twin range
  __shared__ int     sNext;     // the CTA's next item
  __shared__ int     sThinc;    // entries of the THINC list
  // faces that take the reference arithmetic, and the ghosted cells with a
  // primitive out of range (one bit each)
  using FaceId = typename std::conditional<B == 8, unsigned char, short>::type;
  constexpr int       NW = (GG + 31) / 32;
  __shared__ int      sCold;
  __shared__ FaceId   sFace[2 * NFF];
  __shared__ unsigned sBad[NW];
  const int          tid = threadIdx.x;
  const PhysParams & P = a.p;
  auto               item_block = [&](int i) {
    const int w = i < n_full ? i : n_full + ((i - n_full) >> split);
    return a.work ? a.work[w] : w;
  };
  if (tid == 0)
    sThinc = sCold = 0;
  if (tid < NW)
    sBad[tid] = 0u;
  __syncthreads();

  for (int iw = blockIdx.x; iw < n_items;)
  {
    const int    n = item_block(iw);
    const int    ty = K::SPLIT && iw >= n_full ? B >> split : B;
    const int    y0 = K::SPLIT && iw >= n_full ? ((iw - n_full) & ((1 << split) - 1)) * ty : 0;
    const int    ncell = B * ty;
    const int    cx0 = a.m.coord[n * 3 + 0], cy0 = a.m.coord[n * 3 + 1];
    // the next item is claimed now (the ticket's latency hides behind the gather)
    const int    next_v = tid == 10 ? claim_next(a, iw, n_items) : 0;
    // coarse/fine slots: loaded now, stored to shared memory at the end of the gather
    int slot_v = -1;
    if (a.m.reflux_slot && tid < 8)
      slot_v = tid < 4 ? a.m.reflux_slot[n * 4 + tid] : a.m.defer_slot[n * 4 + tid - 4];
    if (tid == 8 || tid == 9)
      slot_v = a.fill_twins ? a.m.twin_first[n + tid - 8] : 0;
    const int    ins = a.m.inst ? a.m.inst[n] : 0;
    const double dx = P.level_dx[a.m.level[n]];
    double       dtdx = a.dt[ins];
    // a value left the fast form's range (per thread until the next barrier,
    // then for the whole CTA)
    bool cold = x64_raw_bad(dtdx) || x64_raw_bad(dx);
    {
      const double q = div64(dtdx, dx, cold);
      dtdx = cold ? div_cold64(dtdx, dx) : q;
    }

    // ---------------- phase 1: own cells + halo -> primitives (the own cell is
    // the first item of the threads that have one, the others start on the
    // halo; one copy of the conversion)
    const bool     owner = tid < ncell;
    const int      ci = tid % B, cj = tid / B;
    const double * ublock = a.U + (size_t)n * H::NV * NC;
    const double * own = ublock + B * y0 + tid;
    const int      nhalo = 4 * G + 4 * ty;
    for (int it = owner ? -1 : 0, h = owner ? tid + NT - ncell : tid - ncell; it < 0 || h < nhalo; ++it)
    {
      double u[H::NV];
      int    gx = ci, gy = cj;
      if (it >= 0)
      {
        halo_coords_tile<B>(h, ty, gx, gy);
        h += NT;
      }
      const int by = gy + y0;
      if (gx >= 0 && gx < B && by >= 0 && by < B)
      {
        const double * p = ublock + gx + B * by;
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          u[v] = p[v * NC];
      }
      else if (!gather_ghost_2d<B>(a, n, cx0, cy0, gx, by, u))
      {
        raise_status(a.status, STATUS_MESH);
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          u[v] = ublock[v * NC];
      }
      const int gidx = (gx + 2) + G * (gy + 2);
      double    q[6];
      bool      bad = false;
      prim_fast64<2, false, true, MG>(u, q, P, bad);
      if (bad)
      {
        cold = true;
        State64<2> s;
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          s.v[v] = u[v];
        prim_ref64<2>(s, &P, sQ + gidx, GG);
        bool out = false;
        for (int k = 0; k < 6; ++k)
          out = out || x64_raw_bad(sQ[k * GG + gidx]);
        if (out)
          atomicOr(&sBad[gidx >> 5], 1u << (gidx & 31));
      }
      else
      {
#pragma unroll
        for (int k = 0; k < 6; ++k)
          sQ[k * GG + gidx] = q[k];
      }
    }
    if (tid < 10)
      sSlot[tid] = slot_v;
    if (tid == 10)
      sNext = next_v;
    cold = __syncthreads_or(cold) != 0;
    // the next item of this CTA: its block's cells and table rows into L2
    if (tid < 3 && sNext < n_items)
    {
      const int nn = item_block(sNext);
      if (tid == 0)
        prefetch_l2_range(a.U + (size_t)nn * H::NV * NC, (unsigned)(H::NV * NC * sizeof(double)));
      else if (tid == 1)
        prefetch_l2_line(a.m.nbr + (size_t)nn * 36);
      else
        prefetch_l2_line(a.m.nbr_rel + (size_t)nn * 9);
    }

    // ---------------- phase 2: slopes + Hancock source of the tile's cells,
    // then of the column or row beyond each side
    const bool cold0 = cold;
    for (int h = tid; h < ncell + 2 * ty + 2 * B; h += NT)
    {
      int ri = h % B, rj = h / B;
      if (h >= ncell)
      {
        const int i = h - ncell;
        if (i < 2 * ty)
        {
          ri = i < ty ? -1 : B;
          rj = i < ty ? i : i - ty;
        }
        else
        {
          const int j = i - 2 * ty;
          ri = j % B;
          rj = j < B ? -1 : ty;
        }
      }
      const int r = (ri + 1) + S * (rj + 1), gi = (ri + 2) + G * (rj + 2);
      // In a tile with a value out of range each cell decides by the values
      // that it reads, each face by its two cells, and the faces left over
      // are evaluated from a list, with full warps.  A flow that started at
      // rest holds velocities that fall off to 1e-323 ahead of the waves:
      // 14 % of the shock-bubble's blocks, a few columns of cells in each
      // (431k cells after 5, 20 and 300 steps: 430, 490, 487 -> 364, 395, 391
      // us against the reference arithmetic for the whole tile; 331 us
      // without such values; 383 -> 385 us for 486k cells that have none).
      auto out = [&](int g) { return (sBad[g >> 5] >> (g & 31)) & 1u; };
      bool bad = cold0 && (x64_raw_bad(dtdx) || (out(gi) | out(gi - 1) | out(gi + 1) | out(gi - G) | out(gi + G)) != 0u);
      if (!bad)
        bad = hancock_fast64<B, MG>(sQ, sRec, gi, r, dtdx, P);
      if (bad)
      {
        cold = true;
        hancock_cold64<B>(sQ, sRec, gi, r, dtdx, &P);
        sRec[15 * SS + r] = bad_cell64();
      }
    }
    // the interface cells of the THINC reconstruction
    if (P.thinc != 0)
    {
      for (int i = tid; i < (B + 2) * ty + B * (ty + 2); i += NT)
      {
        int dir, tx, tj;
        thinc_cell<B>(i, ty, dir, tx, tj);
        const double * A = sQ + 5 * GG + (tx + 2) + G * (tj + 2);
        const int      o = dir == 0 ? 1 : G;
        if (thinc_cell64(A[0], A[-o], A[o], P))
          sList[atomicAdd(&sThinc, 1)] = (short)i;
        else
          sAF[i] = sAF[K::NTH + i] = thinc_none64();
      }
    }
    cold = __syncthreads_or(cold) != 0;
    if (P.thinc != 0 && sThinc > 0)
    {
      for (int i = tid; i < sThinc; i += NT)
        cold |= thinc_eval2<B>(sQ, sRec, sAF, sList[i], ty, P);
      cold = __syncthreads_or(cold) != 0;
    }

    // ---------------- phase 3: faces (X then Y) -> HLLC -> shared fluxes
    const bool cold1 = cold;
    const int  nfx = (B + 1) * ty, nf = nfx + B * (ty + 1);
    for (int f = tid; f < nf; f += NT)
    {
      const int dir = f < nfx ? 0 : 1, ff = f - dir * nfx;
      double *  sF = dir == 0 ? sFx : sFy;
      if (face_flux_fast64<B, MG>(sQ, sRec, sAF, sF, ty, dir, ff, cold1, dtdx, P))
      {
        cold = true;
        sFace[atomicAdd(&sCold, 1)] = (FaceId)f;
      }
    }
    // the own cell's state again (an L2 hit, in flight while the CTA waits at
    // the barrier; held from the gather it cost 16 registers)
    double uown[H::NV];
    if (owner)
    {
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
        uown[v] = __ldcg(own + v * NC);
    }
    cold = __syncthreads_or(cold) != 0;
    if (cold)
    {
      for (int i = tid; i < sCold; i += NT)
      {
        const int f = sFace[i], dir = f < nfx ? 0 : 1;
        face_flux_cold64<B>(sQ, sRec, dir == 0 ? sFx : sFy, dir, f - dir * nfx, dtdx, &P);
      }
      __syncthreads();
      if (tid == 0)
        sCold = 0;
      if (tid < NW)
        sBad[tid] = 0u;
    }
    if (tid == 0)
      sThinc = 0; // (read before the barrier above, used again after the next)

    // ---------------- publish coarse/fine records (AMR only)
    if (a.m.reflux_slot && tid < B)
    {
#pragma unroll
      for (int face = 0; face < 4; ++face)
      {
        // the face's cells in the tile: along x faces one per row, along y
        // faces all when the face belongs to the tile
        const int  dir = face >> 1, side = face & 1;
        const bool here = dir == 0 ? tid >= y0 && tid < y0 + ty : (side ? y0 + ty == B : y0 == 0);
        const int  rs = sSlot[face];
        if (rs >= 0 && here)
        {
          // fine block face next to a coarser neighbour: publish its B face fluxes
          const int      idx = dir == 0 ? (side ? B : 0) + (B + 1) * (tid - y0) : tid + B * (side ? ty : 0);
          const double * src = dir == 0 ? sFx : sFy;
          double *       dst = a.reflux_buf + ((size_t)rs * B + tid) * 8;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            dst[k] = src[k * NFF + idx];
        }
        const int ds = sSlot[4 + face];
        if (ds >= 0 && here)
        {
          // coarse cell next to a finer face: save its four own face fluxes
          const int x = dir == 0 ? (side ? B - 1 : 0) : tid;
          const int y = (dir == 0 ? tid : (side ? B - 1 : 0)) - y0;
          double *  dst = a.defer_buf + ((size_t)ds * B + tid) * 32;
          const int fxl = x + (B + 1) * y, fyl = x + B * y;
#pragma unroll
          for (int k = 0; k < 8; ++k)
          {
            dst[0 * 8 + k] = sFx[k * NFF + fxl];
            dst[1 * 8 + k] = sFx[k * NFF + fxl + 1];
            dst[2 * 8 + k] = sFy[k * NFF + fyl];
            dst[3 * 8 + k] = sFy[k * NFF + fyl + B];
          }
        }
      }
    }

    // ---------------- phase 4: update of the owned cell
    bool deferred = false;
    if (a.m.defer_slot)
    {
      const int * dsl = sSlot + 4;
      const int   by = cj + y0;
      deferred = (ci == 0 && dsl[0] >= 0) || (ci == B - 1 && dsl[1] >= 0) || (by == 0 && dsl[2] >= 0) || (by == B - 1 && dsl[3] >= 0);
    }
    double m_inv = 0.0;
    double u2[H::NV];
    if (owner && !deferred)
    {
      double * out = a.U2 + (size_t)n * H::NV * NC + B * y0 + tid;
      bool     bad = cold;
      if (!bad)
        m_inv = update_fast64<B, MG>(uown, u2, sFx, sFy, ci, cj, dx, P, a.invdt != nullptr, bad);
      if (bad)
      {
        State64<2> st;
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          st.v[v] = uown[v];
        m_inv = update_cold64<B>(st, out, sFx, sFy, ci, cj, dx, &P, a.invdt != nullptr);
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
    else
    {
#pragma unroll
      for (int v = 0; v < H::NV; ++v)
        u2[v] = uown[v]; // the reflux pass finishes the cell (and its twin cells)
    }
    if (sSlot[9] > sSlot[8])
    {
      // the solver loop's boundary fill of the outside blocks mirroring this
      // block (FillOutside: the last applicable face's copy rule), from the
      // tile's new state staged in the (now free) slope area
      double * sTw = sRec;
      if (owner)
      {
#pragma unroll
        for (int v = 0; v < H::NV; ++v)
          sTw[v * NC + tid] = u2[v];
      }
      __syncthreads();
      for (int t = sSlot[8]; t < sSlot[9]; ++t)
      {
        const int e = a.m.twin_list[t];
        const int o = e >> 3, face = e & 7, dir = face >> 1, bc = P.bc[face];
        const int edge = (face & 1) ? B - 1 : 0;
        for (int c = tid; c < NC; c += NT)
        {
          const int x = c % B, y = c / B;
          const int sx = dir == 0 ? (bc == 2 ? edge : B - 1 - x) : x;
          const int sy = (dir == 1 ? (bc == 2 ? edge : B - 1 - y) : y) - y0;
          if (sy < 0 || sy >= ty)
            continue; // a cell of another tile
          const double * src = sTw + sx + B * sy;
          double *       dst = a.U2 + (size_t)o * H::NV * NC + c;
#pragma unroll
          for (int v = 0; v < H::NV; ++v)
          {
            const double val = src[v * NC];
            dst[v * NC] = (bc == 3 && v == H::IU + dir) ? neg64(val) : val;
          }
        }
      }
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
    const int next = sNext; // read before the barrier: the next item's claim overwrites it
    __syncthreads();
    iw = next;
  }
}

} // namespace g5
