// g5_fp64_2d.cu — FP64 instantiations of the 2D step (--fmad=false, as
// g5_fp64.cu).
#include <algorithm>

#include "g5_fp64_case.h"
#include "g5_launch.h"
#include "g5_step2d.cuh"
#include "g5_step2d_f64.cuh"

namespace g5
{

// the step kernel of a form: the fast one's, or the reference arithmetic's
template <int B, int STIFF>
struct Step2dLaunch
{
  static constexpr int NT = STIFF != REF64 ? Step2D64<B>::NT : Step2DTraits<B, false>::NT;
  static constexpr bool SPLIT = STIFF != REF64 && Step2D64<B>::SPLIT;
  static size_t
  smem(bool thinc)
  {
    return STIFF != REF64 ? Step2D64<B>::smem_bytes + (thinc ? Step2D64<B>::smem_thinc : 0) : Step2DTraits<B, false>::smem_bytes;
  }
  static auto
  kernel()
  {
    if constexpr (STIFF != REF64)
      return step2d_fast64_kernel<B, STIFF == FASTMG64>;
    else
      return step2d_kernel<B, false>;
  }
};

template <int B, int STIFF>
static int
occupancy2d(bool thinc)
{
  using K = Step2dLaunch<B, STIFF>;
  cudaFuncSetAttribute(K::kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem(true));
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, K::kernel(), K::NT, K::smem(thinc));
  return occ;
}

template <int B, int STIFF>
static cudaError_t
launch_step2d(const StepArgs & a, int ctas_per_sm, cudaStream_t s, int * launches)
{
  using K = Step2dLaunch<B, STIFF>;
  static const int occs[2] = { std::max(1, occupancy2d<B, STIFF>(false)), std::max(1, occupancy2d<B, STIFF>(true)) };
  const int        occ = occs[a.p.thinc != 0];
  const int        per_sm = (ctas_per_sm > 0 && ctas_per_sm < occ) ? ctas_per_sm : occ;
  const int        slots = num_sms() * per_sm, nwalk = step_count(a);
  // a last round of blocks that fills at most half of the resident CTAs is
  // taken in halves (fuller ones gain nothing: 185 blocks on 304 CTAs), in
  // quarters when they leave SMs without a tile (8 to 38 blocks: 31 -> 29 us)
  const int last = nwalk % slots;
  const int split = !K::SPLIT || last == 0 || 2 * last > slots ? 0 : (4 * last <= num_sms() ? 2 : 1);
  const int n_full = split ? nwalk - last : nwalk;
  const int n_items = n_full + ((nwalk - n_full) << split);
  const int grid = std::min(slots, n_items);
  cudaError_t e = cudaSuccess;
  if (grid >= 1)
  {
    if constexpr (STIFF != REF64)
      K::kernel()<<<grid, K::NT, K::smem(a.p.thinc != 0), s>>>(a, n_full, n_items, split);
    else
      K::kernel()<<<grid, K::NT, K::smem(false), s>>>(a);
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
