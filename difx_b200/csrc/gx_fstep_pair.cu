// Host side of the paired-band F-step (gx_fstep_pair.cuh): how the time samples
// are decoded, blocks per CTA, phase-cal fusion, dispatch.
#include "gx_fstep_pair.cuh"

namespace gx {

static PairDecode pair_decode(const DevJob &J)
{
  PairDecode D{};
  const int band = J.nbits * (J.cplx ? 2 : 1);
  const bool pairs = J.nbands % 2 == 0;   // else each band by itself, two blocks at a time
  D.nfields = pairs ? J.nbands / 2 : J.nbands;
  D.width = pairs ? 2 * band : band;
  D.ts_bits = J.nbands * band;
  // whole columns where the time samples and their frames keep the alignment
  // (station buffers start at a word: blockparams_kernel reads their headers so)
  const bool words = D.ts_bits % 32 == 0 && 32 % D.width == 0 && J.framebytes % 4 == 0;
  const bool narrow = (D.ts_bits == 16 || D.ts_bits == 8) && J.framebytes % 4 == 0;
  D.load = pairs && (words || narrow);
  D.ncol = !D.load ? D.nfields : words ? D.ts_bits / 32 : 1;
  D.ppc = D.nfields / D.ncol;
  D.kind = (!J.cplx && J.nbits <= 2) ? 0 : (J.nbits == 8 && J.lut_offset == kCodeOffset) ? 1 : 2;
  D.scale = D.kind == 1 ? (float)(1.0 / J.lut_div) : 1.0f;
  return D;
}

// Whether the kernel takes this job: transforms of 128 to 8192 points, linear
// or post-F fringe rotation (the quadratic order's rotator is a full table).
bool fstep_pair_eligible(const DevJob &J)
{
  return J.fftlen >= 128 && J.fftlen <= 8192 && J.fringe_order != 2;
}

int fstep_pair_groups(const DevJob &J)
{
  const int NT = J.fftlen / 16;
  return NT >= 256 ? 1 : 256 / NT;
}

// Units of work (FFT blocks, or two of them) per group and CTA: the fewest rounds of two CTAs on each of 148
// SMs (one at 8192 points), counted in blocks, with a fifth of a block for a
// CTA's start (twiddles, station constants, first samples).
static int pair_items(const DevJob &J, int nunit)
{
  if (J.sb_items > 0) return J.sb_items;
  const int G = fstep_pair_groups(J);
  const long long slots = J.fftlen > 4096 ? 148 : 296;
  int best = 1;
  double cost = 1e30;
  for (int items = 1; items <= 8; items++) {
    const long long ctas = (long long)((nunit + items * G - 1) / (items * G)) * J.nstations;
    const double c = (double)((ctas + slots - 1) / slots) * (items + 0.2);
    if (c < cost * 0.999) {
      cost = c;
      best = items;
    }
  }
  return best;
}

// Whether the kernel can form the phase-cal sums of pf for this job and
// launch: bins dividing the threads of a transform, one slot per group.
static bool fstep_pair_pcal_fits(const DevJob &J, const PcalFuse &pf, int nunit, int items)
{
  const int NT = J.fftlen / 16, G = fstep_pair_groups(J);
  return pf.partial && pf.first && pf.nbins > 0 && pf.nbins <= NT && NT % pf.nbins == 0 &&
         (long long)((nunit + items * G - 1) / (items * G)) * G <= pf.slots;
}

cudaError_t fstep_pair_launch(const DevJob &J, const DevStation *stations, const SubintArrays &S, int nblk,
                              const BlockParam *bp, float2 *spec, cudaStream_t st, const PcalFuse *pf, bool *pcal_done)
{
  const bool one = J.nbands % 2 != 0;
  const int nunit = one ? (nblk + 1) / 2 : nblk;
  int items = pair_items(J, nunit);
  bool pc = false;
  if (pf) {
    // as many units per group as the slots need (the tuner's choice stands)
    int most = items;
    if (J.sb_items <= 0)
      while (most < 64 && !fstep_pair_pcal_fits(J, *pf, nunit, most)) most++;
    pc = fstep_pair_pcal_fits(J, *pf, nunit, most);
    if (pc) items = most;
  }
  const PcalFuse pfv = pc ? *pf : PcalFuse{};
  if (pcal_done) *pcal_done = pc;
  auto *go = one ? (pc ? pr::launch_one_pc : pr::launch_one)
                 : pc ? (J.cplx ? pr::launch_cplx_pc : pr::launch_real_pc) : (J.cplx ? pr::launch_cplx : pr::launch_real);
  return go(J, stations, S, nblk, items, pair_decode(J), bp, spec, pfv, st);
}

}  // namespace gx
