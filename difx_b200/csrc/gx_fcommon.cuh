// Device helpers shared by the F-step kernels (gx_fstep.cu, gx_fstep_pair.cuh):
// complex products, the per-block rotator table entries (FP64 phases, FP32
// sincos; mode.cpp:882-955, 1029-1122) and group barriers.
#pragma once
#include <cstdint>
#include "gx_dev.h"

namespace gx {

#define GX_TWO_PI 6.283185307179586476925286766559

__device__ __forceinline__ float2 cmul_exact(float2 a, float2 b)
{
  // no contraction: same rounding as the reference's separate multiplies/adds
  float2 r;
  r.x = __fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y));
  r.y = __fadd_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x));
  return r;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// cos and sin of a number of turns (below 2^51): the whole ones removed in
// FP64, the rest in FP32 half turns.
__device__ __forceinline__ float2 unit(double turns)
{
  const double whole = (turns + 6755399441055744.0) - 6755399441055744.0;
  float sn, cs;
  sincospif((float)(2.0 * (turns - whole)), &sn, &cs);
  return make_float2(cs, sn);
}

// Fringe-rotator table entry e of local freq fi, stride Sd, nfr steps: e < Sd ->
// sub[e], else step[e - Sd] (mode.cpp:882-955: FP64 phases, FP32 argument,
// sincos).  The transform length is a power of two: its reciprocal is exact.
__device__ __forceinline__ float2 fringe_entry(const DevJob &J, const DevStation &st, int fi, int e,
                                               const BlockParam &P, int Sd, int nfr)
{
  if (J.fringe_order == 0) return make_float2(1.0f, 0.0f);   // post-F: no rotation before the FFT
  const double lofreq = st.lofreq[fi];
  const double looffset = st.looff[fi];
  const bool looff = (looffset > 0.0 || looffset < 0.0);
  double ph;
  if (e < Sd) {
    double x = ((double)e * J.inv_fftlen) * P.a;
    x += P.b;
    ph = x * lofreq;
    if (st.fractional_lo) ph += (lofreq - (int)lofreq) * (double)P.integerdelay;
    if (looff) {
      ph += ((e * J.sampletime) / 1e6) * -looffset;
      ph += -looffset * P.fracwalltime;
      double fl = fabs(looffset) - (int)fabs(looffset);
      const bool isfrac = fl > (double)0.000000001f;
      if (looffset < 0) fl = -fl;
      if (isfrac) ph += -fl * P.intwalltime;
    }
  } else if (e < Sd + nfr) {
    const int j = e - Sd;
    const double xoff = (double)(j * Sd) * J.inv_fftlen;
    // quadratic: stepxoff b + stepxoff^2 a (mode.cpp:813-819)
    const double x = J.fringe_order == 2 ? xoff * P.qb + (xoff * xoff) * P.qa : xoff * P.a;
    ph = x * lofreq;
    if (looff) ph += ((j * Sd * J.sampletime) / 1e6) * -looffset;
  } else {
    // quadratic only: the per-stride phase step of sub entry k (mode.cpp:810-812)
    const int k = e - Sd - nfr;
    const double x = ((double)k * J.inv_fftlen) * (2 * P.qa * ((double)Sd * J.inv_fftlen));
    ph = x * lofreq;
  }
  return unit(-ph);
}

// The pre-F linear rotator's phase over a block as a line: turns at sample 0
// (whole delays dropped as the reference does) and per sample, LO offset
// included (mode.cpp:882-955); post-F: no rotation before the FFT.
struct FringeLine {
  double at0, slope;
};
__device__ __forceinline__ FringeLine fringe_line(const DevJob &J, const DevStation &st, int fi, const BlockParam &P)
{
  FringeLine f{0.0, 0.0};
  if (J.fringe_order == 0) return f;
  const double lofreq = st.lofreq[fi], looffset = st.looff[fi];
  f.at0 = P.b * lofreq;
  f.slope = P.a * J.inv_fftlen * lofreq;
  if (st.fractional_lo) f.at0 += (lofreq - (int)lofreq) * (double)P.integerdelay;
  if (looffset != 0.0) {
    f.slope -= J.sampletime * 1e-6 * looffset;
    f.at0 -= looffset * P.fracwalltime;
    double fl = fabs(looffset) - (int)fabs(looffset);
    const bool isfrac = fl > (double)0.000000001f;
    if (looffset < 0) fl = -fl;
    if (isfrac) f.at0 -= fl * P.intwalltime;
  }
  return f;
}

// Fractional-sample angle per us (mode.cpp:1029-1122): of sub entry e, or of
// step e (of `half` steps of Sd channels; a lower sideband's run up to zero).
// The channel count is a power of two: its reciprocal is exact.
__device__ __forceinline__ float frac_freq(const DevJob &J, int e, bool step, bool lsb, int Sd, int half)
{
  if (!step) return (float)((GX_TWO_PI * (e) * J.bw) * J.inv_nchan);
  return lsb ? (float)((-GX_TWO_PI * ((half - e) * Sd) * J.bw) * J.inv_nchan)
             : (float)((GX_TWO_PI * e * Sd * J.bw) * J.inv_nchan);
}

// The fractional sample (us) that a local freq's polarisation set ps (0: A,
// 1: B) is corrected by, clock offsets included.
__device__ __forceinline__ float frac_val(const DevStation &st, int fi, int ps, const BlockParam &P)
{
  const double sgn = ps == 0 ? 1.0 : -1.0;
  return (float)((double)P.fracsampleerror - st.clk[fi] + sgn * st.clkdelta[fi] * 0.5);
}

// Post-F fringe rotation (and LO offset) at the block centre, added to the
// sub entries' arguments for both polarisation sets (mode.cpp:1038-1049, 1085-1096).
__device__ __forceinline__ float frac_post(const DevJob &J, const DevStation &st, int fi, const BlockParam &P)
{
  if (J.fringe_order != 0) return 0.f;
  const double lofreq = st.lofreq[fi];
  double ph = P.b * lofreq;
  if (st.fractional_lo) ph += P.integerdelay * (lofreq - (int)lofreq);
  ph -= ((double)P.intwalltime + P.fracwalltime) * st.looff[fi];
  return (float)(-GX_TWO_PI * (ph - (int)ph));
}

// Fractional-sample rotator entry e of local freq fi: e < Sd -> sub[e], else step[e - Sd].
__device__ __forceinline__ float2 frac_entry(const DevJob &J, const DevStation &st, int fi, int ps, int e,
                                             const BlockParam &P, int Sd, int half)
{
  const bool step = e >= Sd;
  float arg = __fmul_rn(frac_freq(J, step ? e - Sd : e, step, st.lsb[fi], Sd, half), frac_val(st, fi, ps, P));
  if (!step) arg = __fadd_rn(arg, frac_post(J, st, fi, P));
  float sn, cs;
  sincosf(arg, &sn, &cs);
  return make_float2(cs, sn);
}

template <int NT, int CTA>
__device__ __forceinline__ void group_sync(int g)
{
  if constexpr (NT == 32) __syncwarp();
  else if constexpr (NT == CTA) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(NT) : "memory");
}

}  // namespace gx
