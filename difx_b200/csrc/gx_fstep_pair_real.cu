// Station-pair F-step kernels (gx_fstep_pair.cuh) of real data.
#include "gx_fstep_pair.cuh"

namespace gx {
namespace pr {

cudaError_t launch_real(GX_PAIR_ARGS)
{
  return launch<0, false, false>(J, stations, S, nblk, items, D, bp, spec, pf, st);
}

}  // namespace pr
}  // namespace gx
