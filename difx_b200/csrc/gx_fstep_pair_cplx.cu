// Station-pair F-step kernels (gx_fstep_pair.cuh) of complex data.
#include "gx_fstep_pair.cuh"

namespace gx {
namespace pr {

cudaError_t launch_cplx(GX_PAIR_ARGS)
{
  return launch<1, false, false>(J, stations, S, nblk, items, D, bp, spec, pf, st);
}

}  // namespace pr
}  // namespace gx
