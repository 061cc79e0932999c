// g5_fp64_2d.cu — FP64 instantiations of the 2D step (--fmad=false, as
// g5_fp64.cu).
#include <algorithm>

#include "g5_fp64_case.h"
#include "g5_launch.h"
#include "g5_step2d.cuh"

namespace g5
{

template <int B, int STIFF>
static int
occupancy2d(bool thinc)
{
  using T = Step2DTraits<B, false>;
  const size_t smem = T::smem_bytes + (thinc ? T::smem_thinc : 0);
  cudaFuncSetAttribute(step2d_kernel<B, false, false, STIFF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(T::smem_bytes + T::smem_thinc));
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, step2d_kernel<B, false, false, STIFF>, T::NT, smem);
  return occ;
}

template <int B, int STIFF>
static cudaError_t
launch_step2d(const StepArgs & a, int ctas_per_sm, cudaStream_t s, int * launches)
{
  using T = Step2DTraits<B, false>;
  static const int occs[2] = { std::max(1, occupancy2d<B, STIFF>(false)), std::max(1, occupancy2d<B, STIFF>(true)) };
  const int        occ = occs[a.p.thinc != 0];
  const int        per_sm = (ctas_per_sm > 0 && ctas_per_sm < occ) ? ctas_per_sm : occ;
  int              grid = num_sms() * per_sm;
  if (grid > step_count(a))
    grid = step_count(a);
  cudaError_t e = cudaSuccess;
  if (grid >= 1)
  {
    step2d_kernel<B, false, false, STIFF><<<grid, T::NT, T::smem_bytes + (a.p.thinc != 0 ? T::smem_thinc : 0), s>>>(a);
    ++*launches;
    e = cudaGetLastError();
    if (e != cudaSuccess)
      return e;
  }
  if (a.m.n_defer > 0)
  {
    const int n = a.m.n_defer * B;
    reflux2d_kernel<B, false><<<(n + 31) / 32, 32, 0, s>>>(a);
    ++*launches;
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t
launch_step2d_fp64(int b, const StepArgs & a, int ctas_per_sm, cudaStream_t s, int * launches)
{
  if (b == 16)
    return launch_case64(a.p, [&](auto k) { return launch_step2d<16, k.value>(a, ctas_per_sm, s, launches); });
  if (b == 8)
    return launch_case64(a.p, [&](auto k) { return launch_step2d<8, k.value>(a, ctas_per_sm, s, launches); });
  return cudaErrorInvalidValue;
}

int
step_max_ctas_per_sm_fp64_2d(int b)
{
  if (b == 16)
    return std::min({ occupancy2d<16, FAST64>(true), occupancy2d<16, FASTMG64>(true), occupancy2d<16, REF64>(true) });
  if (b == 8)
    return std::min({ occupancy2d<8, FAST64>(true), occupancy2d<8, FASTMG64>(true), occupancy2d<8, REF64>(true) });
  return 0;
}

} // namespace g5
