// g5_fp64.cu — FP64 instantiations beside the steps (g5_fp64_2d.cu,
// g5_fp64_3d.cu) and the dispatch of every FP64 step.  Built with --fmad=false so that every
// product and sum is rounded separately, as in the reference's arithmetic.
#include <algorithm>

#include "g5_aux.cuh"
#include "g5_fp64_case.h"
#include "g5_launch.h"
#include "g5_prolong.cuh"

namespace g5
{

bool
step_supported(int dim, int b)
{
  return (dim == 2 && (b == 8 || b == 16)) || (dim == 3 && b == 8);
}

template <int DIM, int B, int MODE>
static cudaError_t
prolong_t(const StepArgs & a, cudaStream_t s, int * launches)
{
  using T = ProlongTraits<DIM, B, MODE>;
  static bool configured = false;
  if (!configured)
  {
    const cudaError_t e = cudaFuncSetAttribute(prolong_kernel<DIM, B, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem_bytes);
    if (e != cudaSuccess)
      return e;
    configured = true;
  }
  int grid = num_sms() * 8;
  if (grid > step_count(a))
    grid = step_count(a);
  if (grid < 1)
    return cudaSuccess;
  prolong_kernel<DIM, B, MODE><<<grid, T::NT, T::smem_bytes, s>>>(a);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t
launch_prolong(int dim, int b, const StepArgs & a, cudaStream_t s, int * launches)
{
  if (!a.m.pg)
    return cudaSuccess;
  const int mode = a.p.prolong;
  if (dim == 2 && b == 16)
    return mode == 1 ? prolong_t<2, 16, 1>(a, s, launches)
         : mode == 2 ? prolong_t<2, 16, 2>(a, s, launches)
         : mode == 3 ? prolong_t<2, 16, 3>(a, s, launches)
                     : cudaErrorInvalidValue;
  if (dim == 2 && b == 8)
    return mode == 1 ? prolong_t<2, 8, 1>(a, s, launches)
         : mode == 2 ? prolong_t<2, 8, 2>(a, s, launches)
         : mode == 3 ? prolong_t<2, 8, 3>(a, s, launches)
                     : cudaErrorInvalidValue;
  if (dim == 3 && b == 8)
    return mode == 1 ? prolong_t<3, 8, 1>(a, s, launches)
         : mode == 2 ? prolong_t<3, 8, 2>(a, s, launches)
         : mode == 3 ? prolong_t<3, 8, 3>(a, s, launches)
                     : cudaErrorInvalidValue;
  return cudaErrorInvalidValue;
}

template <int DIM, int B, int MODE>
static cudaError_t
refine_t(const double * Uold, double * Unew, const DevMesh & m, const int32_t * list, int n_ref, unsigned int * status, cudaStream_t s)
{
  using T = RefineTraits<DIM, B, MODE>;
  static bool configured = false;
  if (!configured)
  {
    const cudaError_t e = cudaFuncSetAttribute(prolong_refine_kernel<DIM, B, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem_bytes);
    if (e != cudaSuccess)
      return e;
    configured = true;
  }
  int grid = num_sms() * 4;
  if (grid > n_ref)
    grid = n_ref;
  if (grid < 1)
    return cudaSuccess;
  prolong_refine_kernel<DIM, B, MODE><<<grid, T::NT, T::smem_bytes, s>>>(Uold, Unew, m, list, n_ref, status);
  return cudaGetLastError();
}

cudaError_t
launch_remap_prolong(int dim, int b, int mode, const double * Uold, double * Unew, const DevMesh & m, const int32_t * list, int n_ref,
                     unsigned int * status, cudaStream_t s)
{
  if (dim == 2 && b == 16)
    return mode == 1 ? refine_t<2, 16, 1>(Uold, Unew, m, list, n_ref, status, s)
         : mode == 2 ? refine_t<2, 16, 2>(Uold, Unew, m, list, n_ref, status, s)
         : mode == 3 ? refine_t<2, 16, 3>(Uold, Unew, m, list, n_ref, status, s)
                     : cudaErrorInvalidValue;
  if (dim == 2 && b == 8)
    return mode == 1 ? refine_t<2, 8, 1>(Uold, Unew, m, list, n_ref, status, s)
         : mode == 2 ? refine_t<2, 8, 2>(Uold, Unew, m, list, n_ref, status, s)
         : mode == 3 ? refine_t<2, 8, 3>(Uold, Unew, m, list, n_ref, status, s)
                     : cudaErrorInvalidValue;
  if (dim == 3 && b == 8)
    return mode == 1 ? refine_t<3, 8, 1>(Uold, Unew, m, list, n_ref, status, s)
         : mode == 2 ? refine_t<3, 8, 2>(Uold, Unew, m, list, n_ref, status, s)
         : mode == 3 ? refine_t<3, 8, 3>(Uold, Unew, m, list, n_ref, status, s)
                     : cudaErrorInvalidValue;
  return cudaErrorInvalidValue;
}

cudaError_t
launch_step_fp64(int dim, int b, const StepArgs & a, int ctas_per_sm, cudaStream_t s, int * launches)
{
  const cudaError_t e = launch_prolong(dim, b, a, s, launches);
  if (e != cudaSuccess)
    return e;
  if (dim == 2)
    return launch_step2d_fp64(b, a, ctas_per_sm, s, launches);
  if (dim == 3 && b == 8)
    return launch_step3d_fp64(a, ctas_per_sm, s, launches);
  return cudaErrorInvalidValue;
}

int
step_max_ctas_per_sm_fp64(int dim, int b)
{
  return dim == 2 ? step_max_ctas_per_sm_fp64_2d(b) : (dim == 3 && b == 8 ? step_max_ctas_per_sm_fp64_3d() : 0);
}

template <int DIM, int B>
static cudaError_t
fill_outside_t(double * U, const DevMesh & m, const PhysParams & p, cudaStream_t s)
{
  constexpr int NC = (DIM == 2) ? B * B : B * B * B;
  const long    n = (long)m.n_outside * NC;
  if (n == 0)
    return cudaSuccess;
  fill_outside_kernel<DIM, B><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(U, m, p);
  return cudaGetLastError();
}

cudaError_t
launch_fill_outside(int dim, int b, double * U, const DevMesh & m, const PhysParams & p, cudaStream_t s)
{
  if (dim == 2 && b == 16)
    return fill_outside_t<2, 16>(U, m, p, s);
  if (dim == 2 && b == 8)
    return fill_outside_t<2, 8>(U, m, p, s);
  if (dim == 3 && b == 8)
    return fill_outside_t<3, 8>(U, m, p, s);
  return cudaErrorInvalidValue;
}

template <int DIM, int B>
static cudaError_t
inv_dt_t(const double * U, const DevMesh & m, const PhysParams & p, double * invdt, cudaStream_t s)
{
  if (m.n_owned == 0)
    return cudaSuccess;
  int grid = num_sms() * 8;
  if (grid > m.n_owned)
    grid = m.n_owned;
  return launch_case64(p, [&](auto k) {
    inv_dt_kernel<DIM, B, k.value><<<grid, 256, 0, s>>>(U, m, p, invdt);
    return cudaGetLastError();
  });
}

cudaError_t
launch_inv_dt(int dim, int b, const double * U, const DevMesh & m, const PhysParams & p, double * invdt, cudaStream_t s)
{
  if (dim == 2 && b == 16)
    return inv_dt_t<2, 16>(U, m, p, invdt, s);
  if (dim == 2 && b == 8)
    return inv_dt_t<2, 8>(U, m, p, invdt, s);
  if (dim == 3 && b == 8)
    return inv_dt_t<3, 8>(U, m, p, invdt, s);
  return cudaErrorInvalidValue;
}

template <int DIM, int B>
static cudaError_t
rk2_t(const double * U, double * U2, const DevMesh & m, const PhysParams & p, double * invdt, cudaStream_t s)
{
  if (m.n_owned == 0)
    return cudaSuccess;
  int grid = num_sms() * 8;
  if (grid > m.n_owned)
    grid = m.n_owned;
  return launch_case64(p, [&](auto k) {
    rk2_combine_kernel<DIM, B, false, k.value><<<grid, 256, 0, s>>>(U, U2, m, p, invdt);
    return cudaGetLastError();
  });
}

cudaError_t
launch_rk2_combine(int dim, int b, bool mixed, const double * U, double * U2, const DevMesh & m, const PhysParams & p, double * invdt,
                   cudaStream_t s)
{
  if (mixed)
    return launch_rk2_combine_mixed(dim, b, U, U2, m, p, invdt, s);
  if (dim == 2 && b == 16)
    return rk2_t<2, 16>(U, U2, m, p, invdt, s);
  if (dim == 2 && b == 8)
    return rk2_t<2, 8>(U, U2, m, p, invdt, s);
  if (dim == 3 && b == 8)
    return rk2_t<3, 8>(U, U2, m, p, invdt, s);
  return cudaErrorInvalidValue;
}

cudaError_t
launch_dt_update(double * invdt, double * dt, double * dt_hist, int n_inst, double cfl, cudaStream_t s)
{
  dt_update_kernel<<<(n_inst + 127) / 128, 128, 0, s>>>(invdt, dt, dt_hist, n_inst, cfl);
  return cudaGetLastError();
}

template <int DIM, int B>
static cudaError_t
flags_t(const double * U, const DevMesh & m, int ind, double er, double ec, double el, int lmin, int lmax, int8_t * flags, cudaStream_t s)
{
  if (m.n_owned == 0)
    return cudaSuccess;
  int grid = num_sms() * 8;
  if (grid > m.n_owned)
    grid = m.n_owned;
  constexpr int NC = DIM == 2 ? B * B : B * B * B;
  // (negative thresholds keep the general kernel)
  if (ind == 0 && er >= 0.0 && ec >= 0.0)
    gradient_flags_kernel<DIM, B><<<std::min(m.n_owned, num_sms() * (2048 / NC)), NC, 0, s>>>(U, m, er, ec, (float)er, (float)ec, lmin, lmax, flags);
  else
    refine_flags_kernel<DIM, B><<<grid, 256, 0, s>>>(U, m, ind, er, ec, el, lmin, lmax, flags);
  return cudaGetLastError();
}

cudaError_t
launch_refine_flags(int dim, int b, const double * U, const DevMesh & m, int indicator, double er, double ec, double el,
                    int lmin, int lmax, int8_t * flags, cudaStream_t s)
{
  if (dim == 2 && b == 16)
    return flags_t<2, 16>(U, m, indicator, er, ec, el, lmin, lmax, flags, s);
  if (dim == 2 && b == 8)
    return flags_t<2, 8>(U, m, indicator, er, ec, el, lmin, lmax, flags, s);
  if (dim == 3 && b == 8)
    return flags_t<3, 8>(U, m, indicator, er, ec, el, lmin, lmax, flags, s);
  return cudaErrorInvalidValue;
}

template <int DIM, int B>
static cudaError_t
remap_t(const double * Uold, double * Unew, const int8_t * kind, const int32_t * src, int n_new, cudaStream_t s)
{
  if (n_new == 0)
    return cudaSuccess;
  int grid = num_sms() * 8;
  if (grid > n_new)
    grid = n_new;
  remap_kernel<DIM, B><<<grid, 256, 0, s>>>(Uold, Unew, kind, src, n_new);
  return cudaGetLastError();
}

cudaError_t
launch_remap(int dim, int b, const double * Uold, double * Unew, const int8_t * kind, const int32_t * src, int n_new, cudaStream_t s)
{
  if (dim == 2 && b == 16)
    return remap_t<2, 16>(Uold, Unew, kind, src, n_new, s);
  if (dim == 2 && b == 8)
    return remap_t<2, 8>(Uold, Unew, kind, src, n_new, s);
  if (dim == 3 && b == 8)
    return remap_t<3, 8>(Uold, Unew, kind, src, n_new, s);
  return cudaErrorInvalidValue;
}

cudaError_t
launch_defer_info(int dim, const DevMesh & m, const int32_t * codes, int n, int32_t * info, cudaStream_t s)
{
  if (n <= 0)
    return cudaSuccess;
  if (dim == 2)
    defer_info_kernel<2><<<(n + 127) / 128, 128, 0, s>>>(m, codes, n, info);
  else
    defer_info_kernel<3><<<(n + 127) / 128, 128, 0, s>>>(m, codes, n, info);
  return cudaGetLastError();
}

template <int DIM, int B>
static cudaError_t
fields_t(const double * U, double * out, const FieldList & fl, long long stride, long long oct_begin, long long num_octs, const PhysParams & p,
         cudaStream_t s)
{
  constexpr int   NC = DIM == 2 ? B * B : B * B * B;
  const long long total = num_octs * NC;
  if (total <= 0)
    return cudaSuccess;
  const unsigned grid = (unsigned)std::min<long long>((total + 255) / 256, (long long)num_sms() * 16);
  return launch_case64(p, [&](auto k) {
    fields_kernel<DIM, B, k.value><<<grid, 256, 0, s>>>(U, out, fl, stride, oct_begin, num_octs, p);
    return cudaGetLastError();
  });
}

static cudaError_t
launch_fields(int dim, int b, const double * U, double * out, const FieldList & fl, long long stride, long long oct_begin, long long num_octs,
              const PhysParams & p, cudaStream_t s)
{
  if (dim == 2 && b == 16)
    return fields_t<2, 16>(U, out, fl, stride, oct_begin, num_octs, p, s);
  if (dim == 2 && b == 8)
    return fields_t<2, 8>(U, out, fl, stride, oct_begin, num_octs, p, s);
  if (dim == 3 && b == 8)
    return fields_t<3, 8>(U, out, fl, stride, oct_begin, num_octs, p, s);
  return cudaErrorInvalidValue;
}

cudaError_t
launch_derived(int dim, int b, const double * U, double * out, int quantity, long long oct_begin, long long num_octs, const PhysParams & p,
               cudaStream_t s)
{
  // (the quantity's array covers all blocks, out[oct][cell])
  const int nc = dim == 2 ? b * b : b * b * b;
  FieldList fl = {};
  fl.n = 1;
  fl.code[0] = FIELD_DERIVED + quantity;
  fl.need = (1 << quantity) & ~1;
  return launch_fields(dim, b, U, out + oct_begin * nc, fl, 0, oct_begin, num_octs, p, s);
}

cudaError_t
launch_pack_fields(int dim, int b, const double * U, double * out, const int * codes, int n, long long oct_begin, long long num_octs,
                   const PhysParams & p, cudaStream_t s)
{
  if (n < 1 || n > MAX_PACK_FIELDS)
    return cudaErrorInvalidValue;
  FieldList fl = {};
  fl.n = n;
  for (int k = 0; k < n; ++k)
  {
    fl.code[k] = codes[k];
    if (codes[k] > FIELD_DERIVED)
      fl.need |= 1 << (codes[k] - FIELD_DERIVED);
  }
  return launch_fields(dim, b, U, out, fl, num_octs * (dim == 2 ? b * b : b * b * b), oct_begin, num_octs, p, s);
}

} // namespace g5
