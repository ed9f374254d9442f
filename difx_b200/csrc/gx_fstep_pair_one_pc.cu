// Paired-band F-step kernels (gx_fstep_pair.cuh) of one band and two FFT blocks at a time with phase-cal.
#include "gx_fstep_pair.cuh"

namespace gx {
namespace pr {

cudaError_t launch_one_pc(GX_PAIR_ARGS)
{
  return J.cplx ? launch<1, true, true>(J, stations, S, nblk, items, D, bp, spec, pf, st)
                : launch<0, true, true>(J, stations, S, nblk, items, D, bp, spec, pf, st);
}

}  // namespace pr
}  // namespace gx
