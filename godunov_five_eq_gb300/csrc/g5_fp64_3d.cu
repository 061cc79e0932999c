// g5_fp64_3d.cu — FP64 instantiations of the 3D step (--fmad=false, as
// g5_fp64.cu).
#include <algorithm>

#include "g5_fp64_case.h"
#include "g5_launch.h"
#include "g5_step3d.cuh"
#include "g5_step3d_f64.cuh"

namespace g5
{

// the 3D step: the fast form's kernel, or the reference arithmetic's
template <int STIFF>
struct Step3dLaunch
{
  static constexpr int    NT = STIFF != REF64 ? Step3D64::NT : Step3DTraits<false>::NT;
  static constexpr size_t smem_bytes = STIFF != REF64 ? Step3D64::smem_bytes : Step3DTraits<false>::smem_bytes;
  static auto
  kernel()
  {
    if constexpr (STIFF != REF64)
      return step3d_fast64_kernel<STIFF == FASTMG64>;
    else
      return step3d_kernel<false>;
  }
};

template <int STIFF>
static int
occupancy3d()
{
  using K = Step3dLaunch<STIFF>;
  cudaFuncSetAttribute(K::kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem_bytes);
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, K::kernel(), K::NT, K::smem_bytes);
  return occ;
}

template <int STIFF>
static cudaError_t
launch_step3d(const StepArgs & a, int ctas_per_sm, cudaStream_t s, int * launches)
{
  using K = Step3dLaunch<STIFF>;
  static const int occ = std::max(1, occupancy3d<STIFF>());
  const int        per_sm = (ctas_per_sm > 0 && ctas_per_sm < occ) ? ctas_per_sm : occ;
  int              grid = num_sms() * per_sm;
  if (grid > step_count(a))
    grid = step_count(a);
  cudaError_t e = cudaSuccess;
  if (grid >= 1)
  {
    K::kernel()<<<grid, K::NT, K::smem_bytes, s>>>(a);
    ++*launches;
    e = cudaGetLastError();
    if (e != cudaSuccess)
      return e;
  }
  if (a.m.n_defer > 0)
  {
    const int n = a.m.n_defer * 64;
    reflux3d_kernel<false><<<(n + 31) / 32, 32, 0, s>>>(a);
    ++*launches;
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t
launch_step3d_fp64(const StepArgs & a, int ctas_per_sm, cudaStream_t s, int * launches)
{
  return launch_case64(a.p, [&](auto k) { return launch_step3d<k.value>(a, ctas_per_sm, s, launches); });
}

int
step_max_ctas_per_sm_fp64_3d()
{
  return std::min({ occupancy3d<FAST64>(), occupancy3d<FASTMG64>(), occupancy3d<REF64>() });
}

} // namespace g5
