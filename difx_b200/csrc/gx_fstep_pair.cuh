// F-step of two bands at a time: one group of F / 16 threads per (station, FFT
// block) transforms the station's bands in pairs (2p, 2p + 1), each thread
// holding 16 points of both bands as packed FP32 pairs.  With an odd number of
// bands the two lanes are two consecutive blocks of one band instead.
//
// What bounds it.  A 4096-point transform is about 60 FP32 operations and 16
// bytes of shared-memory exchange a sample against 10 bytes of HBM, so the SM's
// issue slots, FMA pipe and shared memory run out before HBM does.  Packing the
// two bands of a pair into f32x2 registers halves the instructions of the
// butterflies and the exchange-address work and, where the bands are the two
// polarisations of one frequency, shares the rotator tables and products: 65
// thread instructions a band sample against 82 of one band at a time.  64 data
// registers a thread leave 16 warps an SM, so what is left is latency (issue
// active 45-60 %, FMA pipe 42-54 %).  F-step times against the kernels it
// replaced, which took one band at a time and built the rotator tables of
// transforms below 512 points once per band (1 B200; the short transforms'
// now in passes of up to 32768 blocks, in passes of 4096 as before in brackets):
//   4 stations, 2-bit, 256 points, 200 ms subint     2.77 -> 0.37 ms (0.59)
//   11 stations, 1-bit, 128 points, 200 ms           5.00 -> 0.73 ms (0.97)
//   16 stations, 2-bit, 512 points, 50 ms            2.13 -> 1.55 ms (1.61)
//   6 stations, INTERLACEDVDIF, 1024 points, 100 ms  1.64 -> 0.75 ms (0.83)
//   64 stations, 8-bit complex, 4096 points, 32 ms   4.03 -> 3.57 ms
//   64 stations, 2-bit, 8192 points, 32 ms           7.25 -> 7.13 ms
//
// An odd band count as pairs, the last band alone in both lanes, transformed that
// band twice and read its samples byte by byte between the decodes; as two
// blocks of a band, with all of a thread's words on their way before the first
// is used, against that and against one band at a time (16 stations, 8 bits,
// F-step times):
//   1 band, real, 2048 points, 4000 blocks     1.44 -> 0.52 ms (one at a time 0.60)
//   1 band, real, 8192 points, 1000 blocks     1.80 -> 0.66 ms (0.60)
//   1 band, complex, 1024 points, 8000 blocks  1.68 -> 0.55 ms (0.73)
//   1 band, complex, 4096 points, 2000 blocks  1.71 -> 0.57 ms (0.72)
//   3 bands, real, 1024 points, 4000 blocks    1.48 -> 0.70 ms (1.07)
//   3 bands, complex, 1024 points, 2000 blocks 1.02 -> 0.43 ms (0.55)
//
// Per pair of bands a group
//   1. decodes its field of 16 time samples held in registers (one 32-bit
//      column of the time sample, loaded once for all the pairs in it and,
//      for the next column or block, while the transform runs; format_vdif.c:66-146),
//   2. rotates them (mode.cpp:1160-1183) with the two-level tables of
//      mode.cpp:882-955, built by the group just before,
//   3. runs the radix-16 passes (layout of gx_fft16.h) with
//      exchanges through shared memory: 16-byte elements, one pad element in
//      sixteen, so that the eight lanes of each 128-byte phase of a store or
//      load touch different banks.  Transforms of up to 512 points live in one
//      warp and synchronise on it alone; 512 and 8192 points are two halves
//      that swap eight bins a thread in place of a third exchange (8192 points:
//      7.67 -> 7.04 ms),
//   4. keeps the half of the bins that real data needs (the last butterflies
//      form only those: u0 + u1 or u0 - u1 by the sideband), applies the
//      fractional-sample correction (mode.cpp:1185-1261) and stores the rows.
// With phase-cal (PC, gx::PcalFuse) the decoded samples of each band are also
// added into their phase-cal bins (mode.cpp:759-774; the implicit-shift
// extractors of pcal.cpp:1032-1222 and 1419-1600).
#pragma once
#include <algorithm>
#include <cstdint>
#include "gx_dev.h"
#include "gx_fcommon.cuh"
#include "gx_fft16.h"

namespace gx {

cudaError_t smem_opt_in(const void *kernel, size_t bytes);

// How a pair's field is found and decoded; the same for every station of a job.
struct PairDecode {
  int nfields;       // band pairs, or bands where the lanes are two blocks of a band
  int width;         // bits of a pair's or band's field
  int ts_bits;       // bits of a time sample
  int ncol, ppc;     // columns loaded per time sample, pairs per column
  int load;          // 1: pairs are read as aligned columns, 0: bytes of the field one by one
  // 0: level pair from a table of 1- or 2-bit real codes, 1: 8-bit codes by arithmetic, 2: level table
  int kind;
  float scale;       // kind 1: level = (code - kCodeOffset) scale, the scale carried by the rotator
};

// The offset of 8-bit codes that kind 1 takes off; symmetric ones (127.5) use the table.
constexpr int kCodeOffset = 128;

namespace pr {

// What the two lanes of a thread's packed values are.
constexpr int kSameBands = 0;   // two bands of one frequency: one set of rotator tables
constexpr int kTwoBands = 1;    // two bands, a set of tables each
constexpr int kTwoBlocks = 2;   // two consecutive FFT blocks of one band, a set of tables each: odd band counts

struct V {
  float2 re, im;     // the two lanes
};

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ V vadd(V a, V b) { return V{r16::add2(a.re, b.re), r16::add2(a.im, b.im)}; }
__device__ __forceinline__ V vsub(V a, V b) { return V{r16::sub2(a.re, b.re), r16::sub2(a.im, b.im)}; }
// a + s b, s = +-1 per lane
__device__ __forceinline__ V vaddsgn(V a, V b, float2 s) { return V{fma2(b.re, s, a.re), fma2(b.im, s, a.im)}; }
// Both lanes by the complex number (wx, wy): packed (four instructions and
// the copies that pair wx, wy and -wy up) or lane by lane (eight).
template <bool PACKED>
__device__ __forceinline__ V vmul(V a, float wx, float wy)
{
  if constexpr (PACKED)
    return V{fma2(a.im, dup(-wy), mul2(a.re, dup(wx))), fma2(a.im, dup(wx), mul2(a.re, dup(wy)))};
  else
    return V{make_float2(a.re.x * wx - a.im.x * wy, a.re.y * wx - a.im.y * wy),
             make_float2(a.re.x * wy + a.im.x * wx, a.re.y * wy + a.im.y * wx)};
}
// W_16^2 = h (1 - i) and W_16^6 = -h (1 + i)
__device__ __forceinline__ V vmul_w2(V a)
{
  const float2 h = dup(0.70710678118654752440f);
  return V{mul2(r16::add2(a.re, a.im), h), mul2(r16::sub2(a.im, a.re), h)};
}
__device__ __forceinline__ V vmul_w6(V a)
{
  const float2 h = dup(0.70710678118654752440f), m = dup(-0.70710678118654752440f);
  return V{mul2(r16::sub2(a.im, a.re), h), mul2(r16::add2(a.re, a.im), m)};
}

// 4-point forward DFT in place, natural order
__device__ __forceinline__ void dft4(V &a, V &b, V &c, V &d)
{
  const V s0 = vadd(a, c), s1 = vsub(a, c), s2 = vadd(b, d), t = vsub(b, d);
  a = vadd(s0, s2);
  c = vsub(s0, s2);
  b = V{r16::add2(s1.re, t.im), r16::sub2(s1.im, t.re)};   // s1 - i t
  d = V{r16::sub2(s1.re, t.im), r16::add2(s1.im, t.re)};   // s1 + i t
}
// The same with c taken as -i c
__device__ __forceinline__ void dft4_mi(V &a, V &b, V &c, V &d)
{
  const V s0{r16::add2(a.re, c.im), r16::sub2(a.im, c.re)}, s1{r16::sub2(a.re, c.im), r16::add2(a.im, c.re)};
  const V s2 = vadd(b, d), t = vsub(b, d);
  a = vadd(s0, s2);
  c = vsub(s0, s2);
  b = V{r16::add2(s1.re, t.im), r16::sub2(s1.im, t.re)};
  d = V{r16::sub2(s1.re, t.im), r16::add2(s1.im, t.re)};
}
// Outputs 0 and 1 (s = +1) or 2 and 3 (s = -1) of the same transform, in a and b
template <bool MI>   // MI: c taken as -i c
__device__ __forceinline__ void dft4_half(V &a, V &b, V c, V d, float2 s)
{
  V s0, s1;
  if constexpr (MI) {
    s0 = V{r16::add2(a.re, c.im), r16::sub2(a.im, c.re)};
    s1 = V{r16::sub2(a.re, c.im), r16::add2(a.im, c.re)};
  } else {
    s0 = vadd(a, c);
    s1 = vsub(a, c);
  }
  const V s2 = vadd(b, d), t = vsub(b, d);
  const float2 ns = make_float2(-s.x, -s.y);
  a = vaddsgn(s0, s2, s);
  b = V{fma2(t.im, s, s1.re), fma2(t.re, ns, s1.im)};
}

// 8-point forward DFT in place, natural order; HALF: outputs 0..3 (s = +1) or
// 4..7 (s = -1) in u[0..3]
template <bool HALF>
__device__ __forceinline__ void dft8(V (&u)[8], float2 s)
{
  dft4(u[0], u[2], u[4], u[6]);
  dft4(u[1], u[3], u[5], u[7]);
  const V o0 = u[1], o1 = vmul_w2(u[3]), o2 = u[5], o3 = vmul_w6(u[7]);   // o2 to be taken times -i
  const V e0 = u[0], e1 = u[2], e2 = u[4], e3 = u[6];
  // W_8^3 = -h (1 + i) = W_16^6
  if constexpr (HALF) {
    u[0] = vaddsgn(e0, o0, s);
    u[1] = vaddsgn(e1, o1, s);
    u[2] = V{fma2(o2.im, s, e2.re), fma2(o2.re, make_float2(-s.x, -s.y), e2.im)};
    u[3] = vaddsgn(e3, o3, s);
  } else {
    u[0] = vadd(e0, o0);
    u[4] = vsub(e0, o0);
    u[1] = vadd(e1, o1);
    u[5] = vsub(e1, o1);
    u[2] = V{r16::add2(e2.re, o2.im), r16::sub2(e2.im, o2.re)};
    u[6] = V{r16::sub2(e2.re, o2.im), r16::add2(e2.im, o2.re)};
    u[3] = vadd(e3, o3);
    u[7] = vsub(e3, o3);
  }
}

// 16-point forward DFT in place, natural order; HALF: outputs 0..7 (s = +1) or
// 8..15 (s = -1) in v[0..7]
template <bool HALF>
__device__ __forceinline__ void dft16(V (&v)[16], float2 s)
{
  const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
#pragma unroll
  for (int n2 = 0; n2 < 4; n2++) dft4(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
  // y[n2][k1] sits at v[4 k1 + n2]; multiply by W16^(n2 k1)
  v[5] = vmul<false>(v[5], c1, -s1);
  v[9] = vmul_w2(v[9]);
  v[13] = vmul<false>(v[13], s1, -c1);
  v[6] = vmul_w2(v[6]);
  // v[10] times W^4 = -i in the butterfly below
  v[14] = vmul_w6(v[14]);
  v[7] = vmul<false>(v[7], s1, -c1);
  v[11] = vmul_w6(v[11]);
  v[15] = vmul<false>(v[15], -c1, s1);
  if constexpr (HALF) {
    V o[8];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
      V a = v[4 * k1], b = v[4 * k1 + 1];
      if (k1 == 2) dft4_half<true>(a, b, v[4 * k1 + 2], v[4 * k1 + 3], s);
      else dft4_half<false>(a, b, v[4 * k1 + 2], v[4 * k1 + 3], s);
      o[k1] = a;
      o[k1 + 4] = b;
    }
#pragma unroll
    for (int t = 0; t < 8; t++) v[t] = o[t];
  } else {
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
      if (k1 == 2) dft4_mi(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
      else dft4(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = a + 1; b < 4; b++) {
        const V t = v[4 * a + b];
        v[4 * a + b] = v[4 * b + a];
        v[4 * b + a] = t;
      }
  }
}

__host__ __device__ constexpr int default_stride(int n)
{
  if (n <= 16) return n;
  int g = 1;
  while ((g + 1) * (g + 1) <= n) g++;
  while (n % g != 0) g--;
  return n / g;
}
__host__ __device__ constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x >> 1); }

// Twiddle rows W^(r m), m < 16, entry m kTwPitch + r: two consecutive r come with
// one 16-byte load, and the pitch (9 x 16 bytes) spreads eight m over the banks.
constexpr int kTwPitch = 18;
constexpr int kTwRow = 16 * kTwPitch;

template <int F, int CPLX>
struct Cfg {
  static constexpr int NT = F / 16;                    // threads per transform
  static constexpr int CTA = NT >= 256 ? NT : 256;
  static constexpr int G = CTA / NT;                   // groups (blocks in flight) per CTA
  static constexpr int N = CPLX ? F : F / 2;           // channels
  static constexpr int L = r16::log16_floor(F);        // radix-16 passes
  static constexpr int R0 = F / r16::pow16(L);         // final radix (1: none)
  // a final radix of 2 (512 and 8192 points): each half of the group transforms
  // the even or the odd samples, and the halves swap half their bins
  static constexpr bool SPLIT = R0 == 2;
  static constexpr int NTS = SPLIT ? NT / 2 : NT;      // threads, points of the transform a thread works in
  static constexpr int FS = NTS * 16;
  // rotator stride: the reference's (calcstridelength, configuration.cpp:37-50)
  // or those threads, so that a thread's samples, and its channels, share a sub entry
  static constexpr int S = default_stride(N) < NTS ? default_stride(N) : NTS;
  static constexpr int LGS = ilog2(S);
  static constexpr int NFR = F / S;                    // fringe steps
  static constexpr int HALF = N / S;                   // fractional-sample steps
  static constexpr int T = 2 * S + NFR + HALF;         // entries of one band's tables
  static constexpr int XB = F + F / 16;                // exchange elements of a group
  static constexpr int FIN = R0 > 1 ? (R0 - 1) * (F / R0) : 0;   // final-pass twiddles: W_F^(r g), g < F / R0
  static constexpr int TBUF = NT > 32 ? 2 : 1;         // table buffers (a CTA barrier apart, or a warp's)
  // 128 registers a thread: 16 warps of two 256-thread CTAs or one of 512
  static constexpr int MINB = CTA > 256 ? 1 : 2;
  static_assert((S & (S - 1)) == 0 && NT % S == 0, "the stride must be a power of two dividing F / 16");
  static_assert(NTS % S == 0, "");
};

template <int F, int CPLX, int LANES>
__host__ __device__ constexpr size_t group_bytes()
{
  using C = Cfg<F, CPLX>;
  return C::XB * sizeof(float4) + (size_t)(C::TBUF * (LANES == kSameBands ? 1 : 2) * C::T) * sizeof(float2) +
         2 * (LANES == kTwoBlocks ? 2 : 1) * sizeof(BlockParam);
}
template <int F, int CPLX, int LANES>
__host__ __device__ constexpr size_t smem_bytes()
{
  using C = Cfg<F, CPLX>;
  return sizeof(float2) * (2 * kTwRow + C::FIN) + (size_t)C::G * group_bytes<F, CPLX, LANES>();
}

// Radix-16 pass of stride 16 (P = 1) or 256 (P = 2): twiddles from the rows
// A: W_256^(r m) and B: W_4096^(r m), m < 16 (W_4096^(r m) for m < 256 is
// B[r][m mod 16] A[r][m / 16]; the whole stride-256 table is 30 KB).
// Real data: packed products; complex data, where the registers are full, lane by
// lane (F-step of 64 stations, 500 blocks: 3.70 against 3.51 ms complex, 7.01
// against 7.19 ms real).
template <int P, bool HALF, bool PACKED>
__device__ __forceinline__ void pass16(V (&v)[16], int j, const float2 *twA, const float2 *twB, float2 s)
{
  const float4 *a = reinterpret_cast<const float4 *>(twA + (P == 1 ? (j & 15) : ((j >> 4) & 15)) * kTwPitch);
  const float4 *b = reinterpret_cast<const float4 *>(twB + (j & 15) * kTwPitch);
#pragma unroll
  for (int r = 0; r < 16; r += 2) {
    float4 w = a[r / 2];   // W^(r m), W^((r + 1) m)
    if constexpr (P == 2) {
      const float4 q = b[r / 2];
      const float2 lo = r ? r16::mul(make_float2(q.x, q.y), make_float2(w.x, w.y)) : make_float2(1.f, 0.f);
      const float2 hi = r16::mul(make_float2(q.z, q.w), make_float2(w.z, w.w));
      w = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    if (r) v[r] = vmul<PACKED>(v[r], w.x, w.y);
    v[r + 1] = vmul<PACKED>(v[r + 1], w.z, w.w);
  }
  dft16<HALF>(v, s);
}

// Final radix-R0 pass (stride F / R0), twiddles W_F^((j + NT mm) r) from fin.
template <int F, int R0, bool HALF, bool PACKED>
__device__ __forceinline__ void final_pass(V (&v)[16], int j, const float2 *fin, float2 s)
{
  constexpr int M = 16 / R0, NT = F / 16, FR = F / R0;
#pragma unroll
  for (int mm = 0; mm < M; mm++) {
    V u[8];
#pragma unroll
    for (int r = 0; r < R0; r++) u[r] = r == 0 ? v[mm] : vmul<PACKED>(v[mm + M * r], fin[(r - 1) * FR + j + NT * mm].x, fin[(r - 1) * FR + j + NT * mm].y);
    if constexpr (R0 == 4) {
      if constexpr (HALF) {
        dft4_half<false>(u[0], u[1], u[2], u[3], s);
        v[mm] = u[0];
        v[mm + M] = u[1];
      } else {
        dft4(u[0], u[1], u[2], u[3]);
#pragma unroll
        for (int r = 0; r < 4; r++) v[mm + M * r] = u[r];
      }
    } else {
      dft8<HALF>(u, s);
#pragma unroll
      for (int r = 0; r < (HALF ? 4 : 8); r++) v[mm + M * r] = u[r];
    }
  }
}

// 16-byte copy global -> shared that completes asynchronously (cp.async, L2 only).
__device__ __forceinline__ void cp_async16(void *sdst, const void *gsrc)
{
  const unsigned int d = (unsigned int)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
// Waits for this thread's outstanding cp.async copies.
__device__ __forceinline__ void cp_async_wait_all()
{
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// The word at p, or 0 without reading it.
__device__ __forceinline__ uint32_t load_if(const void *p, bool pred)
{
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.u32 %0, 0;\n\t@p ld.global.nc.u32 %0, [%1];\n\t}"
               : "=r"(v)
               : "l"(p), "r"((unsigned int)pred));
  return v;
}

template <int NT, int CTA>
__device__ __forceinline__ void sync_group(int g)
{
  if constexpr (NT <= 32) __syncwarp();
  else group_sync<NT, CTA>(g);
}

__device__ __forceinline__ void store16(const V (&v)[16], int j, int Ns, float4 *xb)
{
  const int m = j & (Ns - 1);
  const int p0 = Ns == 1 ? 17 * j : r16::pad((j - m) * 16 + m);
  const int step = Ns == 1 ? 1 : Ns + (Ns >> 4);
#pragma unroll
  for (int r = 0; r < 16; r++) xb[p0 + step * r] = make_float4(v[r].re.x, v[r].re.y, v[r].im.x, v[r].im.y);
}

template <int F>
__device__ __forceinline__ void load16(V (&v)[16], int j, const float4 *xb)
{
  constexpr int NT = F / 16;
  if constexpr (NT % 16 == 0) {
    constexpr int step = NT + NT / 16;
    const int p0 = r16::pad(j);
#pragma unroll
    for (int t = 0; t < 16; t++) {
      const float4 q = xb[p0 + step * t];
      v[t] = V{make_float2(q.x, q.y), make_float2(q.z, q.w)};
    }
  } else {
#pragma unroll
    for (int t = 0; t < 16; t++) {   // NT = 8: two registers' elements per pad element
      const float4 q = xb[j + NT * t + (t >> 1)];
      v[t] = V{make_float2(q.x, q.y), make_float2(q.z, q.w)};
    }
  }
}

// One band's tables: S sub entries of the fringe rotator, its NFR steps, S sub
// entries of the fractional-sample rotator, its HALF steps.  The steps of one
// thread -- index q + (n / S) t, n threads apart in samples or channels -- are
// consecutive (in t), so that two come with one 16-byte load.
template <int N, int S>
__device__ __forceinline__ int step_pos(int x, int per) { return (x & (N / S - 1)) * per + x / (N / S); }

// Builds one band's tables: thread j of the group's NT takes entries j, j + NT,
// ... of the reference's order (mode.cpp:882-955, 1029-1122).  All phases are
// FP64 turns with the whole turns removed, then FP32: the fringe rotator's lie
// on one line over the block, the fractional-sample rotator's are its FP32
// angles.  No branches, so that a thread's entries overlap: one after the
// other their latency was a fifth of a 512-point block's time.  cf: the
// fractional-sample angles per us of the sub entries, then of the upper and of
// the lower sideband's steps.
template <typename C>
__device__ __forceinline__ void put_entries(const DevJob &J, const DevStation &st, int lf, int ps, int j,
                                            const BlockParam &P, float scale, const float *cf, float2 *tab)
{
  const FringeLine fr = fringe_line(J, st, lf, P);
  const float val = frac_val(st, lf, ps, P), post = frac_post(J, st, lf, P);
  const float *cstep = cf + C::S + (st.lsb[lf] ? C::HALF : 0);
  constexpr int K = (C::T + C::NT - 1) / C::NT;
#pragma unroll(K <= 4 ? K : 3)
  for (int k = 0; k < K; k++) {
    const int e = j + C::NT * k;
    if (C::T % C::NT != 0 && e >= C::T) break;
    // e: fringe sub, fringe step, fractional sub, fractional step
    const bool fringe = e < C::S + C::NFR;
    const int i = fringe ? e : e - C::S - C::NFR;
    const bool sub = i < C::S;
    const int x = sub ? i : i - C::S;
    const double line = (sub ? fr.at0 : 0.0) + (double)(sub ? x : x * C::S) * fr.slope;
    const float arg = __fadd_rn(__fmul_rn(sub ? cf[x & (C::S - 1)] : cstep[x & (C::HALF - 1)], val), sub ? post : 0.f);
    const float2 w = unit(fringe ? -line : (double)arg * (1.0 / GX_TWO_PI));
    const float g = fringe && sub ? scale : 1.f;
    const int at = fringe ? (sub ? i : C::S + step_pos<C::NT, C::S>(x, 16))
                          : C::S + C::NFR + (sub ? i : C::S + step_pos<C::NTS, C::S>(x, C::N / C::NTS));
    tab[at] = make_float2(w.x * g, w.y * g);
  }
}

// Pad slot of thread j in the exchange buffer: position 17 k + 16 is never an
// element, so a thread's phase-cal sums park there while the transform runs.
// (m: the thread's first sample; a split group's halves have a buffer each)
template <typename C>
__device__ __forceinline__ int pc_slot(int m)
{
  return C::SPLIT ? (m & 1) * (C::FS + C::FS / 16) + 17 * (m >> 1) + 16 : 17 * m + 16;
}

template <int F, int CPLX, int LANES, bool PC>
__global__ void __launch_bounds__(Cfg<F, CPLX>::CTA, Cfg<F, CPLX>::MINB)
fstep_pair_kernel(const __grid_constant__ DevJob J, const DevStation *__restrict__ stations, SubintArrays S,
                  const BlockParam *__restrict__ bp, int nblk, int blocks_per_group, PairDecode D,
                  float2 *__restrict__ spec, PcalFuse pf)
{
  using C = Cfg<F, CPLX>;
  constexpr int NT = C::NT, CTA = C::CTA, G = C::G, N = C::N, SD = C::S, LGS = C::LGS, T = C::T;
  constexpr bool SAME = LANES == kSameBands;
  constexpr int SETS = SAME ? 1 : 2;
  constexpr int NB = LANES == kTwoBlocks ? 2 : 1;   // blocks of a unit of a group's work
  constexpr bool HALF = !CPLX;
  constexpr int NOUT = CPLX ? 16 : 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float s_lut[256];
  __shared__ float2 s_pl[16];   // level pairs of 1- and 2-bit real codes
  __shared__ float s_cf[SD + 2 * C::HALF];   // fractional-sample angles per us
  const int s = blockIdx.y;
  const int tid = threadIdx.x, g = tid / NT, j = tid % NT;
  // the station's constants are read throughout: a copy in shared memory
  __shared__ __align__(16) DevStation st;
  static_assert(sizeof(DevStation) % 4 == 0 && sizeof(BlockParam) == 80, "copied by words");
  for (int i = tid; i < (int)(sizeof(DevStation) / 4); i += CTA)
    reinterpret_cast<uint32_t *>(&st)[i] = reinterpret_cast<const uint32_t *>(stations + s)[i];
  float2 *twA = reinterpret_cast<float2 *>(smem_raw);
  float2 *twB = twA + kTwRow;
  float2 *fin = twB + kTwRow;
  unsigned char *mine = reinterpret_cast<unsigned char *>(fin + C::FIN) + (size_t)g * group_bytes<F, CPLX, LANES>();
  float4 *xb = reinterpret_cast<float4 *>(mine);
  float2 *tabs = reinterpret_cast<float2 *>(mine + C::XB * sizeof(float4));
  // parameters of the group's current unit of NB blocks and of its next one
  BlockParam *const pbuf = reinterpret_cast<BlockParam *>(tabs + C::TBUF * SETS * T);

  for (int i = tid; i < 256; i += CTA) s_lut[i] = J.lut[i];
  for (int i = tid; i < SD + 2 * C::HALF; i += CTA)
    s_cf[i] = frac_freq(J, i < SD ? i : (i - SD) % C::HALF, i >= SD, i >= SD + C::HALF, SD, C::HALF);
  if (tid < 16) {
    const int m = (1 << J.nbits) - 1;
    s_pl[tid] = make_float2(J.lut[tid & m], J.lut[(tid >> J.nbits) & m]);
  }
  if constexpr (C::L >= 2)
    for (int i = tid; i < 240; i += CTA)
      twA[(i & 15) * kTwPitch + (i >> 4) + 1] = J.twiddle[r16::tw_pass_offset(F, 1) + i];
  if constexpr (C::L >= 3)
    for (int i = tid; i < 240; i += CTA)
      twB[(i & 15) * kTwPitch + (i >> 4) + 1] = J.twiddle[r16::tw_pass_offset(F, 2) + (i >> 4) * 256 + (i & 15)];
  for (int i = tid; i < C::FIN; i += CTA) fin[i] = J.twiddle[r16::tw_final_offset(F) + i];
  __syncthreads();

  const uint8_t *data = S.data[s];
  const int fsamp = J.framesamples, fbytes = J.framebytes;
  const int nunit = (nblk + NB - 1) / NB;
  // phase-cal: as the binning kernels form it
  const int pcfirst = PC ? pf.first[s] : -1;
  const int pcn = PC ? pf.nbins : 1;
  unsigned long long pcs0 = 0;
  if (PC && pcfirst >= 0) {
    const int32_t *ctrl = S.control + (size_t)s * S.controlstride;
    pcs0 = (unsigned long long)(((double)ctrl[1] * 1e9 + (double)ctrl[2]) / (J.sampletime * 1e3) + 0.5);
  }
  float2 *pcout = PC && pcfirst >= 0
                      ? pf.partial + ((size_t)(blockIdx.x * G + g) * pf.nbands_total + pcfirst) * pf.maxbins
                      : nullptr;

  // the half of a split transform, the thread in it, and its first sample (the others NT apart)
  const int h = C::SPLIT ? j / C::NTS : 0, jj = C::SPLIT ? j % C::NTS : j, jb = C::SPLIT ? 2 * jj + h : j;
  float4 *const xh = xb + h * (C::FS + C::FS / 16);
  auto sync_half = [&]() {
    if constexpr (C::SPLIT && C::NTS > 32) asm volatile("bar.sync %0, %1;" ::"r"(h + 1), "r"(C::NTS) : "memory");
    else sync_group<NT, CTA>(g);
  };
  uint32_t raw[16];        // words with the time samples' current column
  int rsh = 0;             // bits below the column (the same for all of a thread's samples)
  unsigned int vmask = 0;  // bit t: sample j + NT t is valid (before any per-band mask)
  unsigned int vmask1 = 0; // the same of a unit's second block
  bool live = false;       // a block of the unit in raw (and the masks) is processed
  const bool fast = NB == 1 && D.load && NT <= fsamp;
  // Copies unit u's parameters into a buffer (completes before the copying
  // threads' cp_async_wait_all; state 0 where there is no such block).
  auto fetch_param = [&](int u, BlockParam *dst) {
    constexpr int kPieces = (int)(sizeof(BlockParam) / 16);
    for (int i = j; i < NB * kPieces; i += NT) {
      if (u * NB + i / kPieces < nblk) cp_async16(reinterpret_cast<char *>(dst) + 16 * i, reinterpret_cast<const char *>(bp + (size_t)s * nblk + u * NB) + 16 * i);
      else reinterpret_cast<uint4 *>(dst)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
  };
  // Loads column col of the samples j + NT t of the block P; samples of invalid
  // frames (and blocks that are not processed) are not read.
  auto load_column = [&](const BlockParam &P, int col) {
    vmask = 0;
    live = P.state != 0;
    if (!live) return;
    const int smp0 = P.nearestsample + jb;
    int q = smp0 / fsamp, r = smp0 - q * fsamp;
    const int nfr = P.nframes;
    const unsigned long long vm = P.validmask;
    if (nfr >= 64 ? vm == ~0ull : vm == ((1ull << nfr) - 1ull)) {
      vmask = 0xFFFFu;
    } else {
      int q1 = q - P.fr0, r1 = r;
#pragma unroll 1
      for (int t = 0; t < 16; t++) {
        vmask |= (unsigned int)((vm >> min(q1, 63)) & 1ull) << t;
        r1 += NT;
        while (r1 >= fsamp) {
          r1 -= fsamp;
          q1++;
        }
      }
    }
    const uint8_t *fr = data + (long long)q * fbytes + 32;
    if (fast) {
      // the aligned words that hold the column; frames and their payloads are
      // whole words, so they end within the frame, and the samples of a thread
      // start at the same bit of theirs
      const int bpts = D.ts_bits >> 3;
      const uint8_t *p = fr + (long long)r * bpts + 4 * col;
      const int adv = NT * bpts, hop = fbytes - fsamp * bpts;   // next frame: past its header
      int left = fsamp - r;
      rsh = 8 * (int)(reinterpret_cast<uintptr_t>(p) & 3);
      p -= rsh >> 3;
#pragma unroll
      for (int t = 0; t < 16; t++) {
        raw[t] = 0;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.u32 %0, 0;\n\t@p ld.global.nc.u32 %0, [%1];\n\t}"
                     : "=r"(raw[t])
                     : "l"(p), "r"((vmask >> t) & 1u));
        p += adv;
        left -= NT;
        if (left <= 0) {
          p += hop;
          left += fsamp;
        }
      }
    }
  };
  // Which of the thread's samples of the block P are valid.
  auto valid_samples = [&](const BlockParam &P) {
    const int nfr = P.nframes, smp0 = P.nearestsample + jb;
    const unsigned long long vm = P.validmask;
    if (P.state == 0) return 0u;
    if (nfr >= 64 ? vm == ~0ull : vm == ((1ull << nfr) - 1ull)) return 0xFFFFu;
    int q = smp0 / fsamp, r = smp0 - q * fsamp;
    unsigned int m = 0;
    q -= P.fr0;
#pragma unroll 1
    for (int t = 0; t < 16; t++) {
      m |= (unsigned int)((vm >> min(q, 63)) & 1ull) << t;
      r += NT;
      while (r >= fsamp) {
        r -= fsamp;
        q++;
      }
    }
    return m;
  };
  // Takes over the unit P: of one block, column col too; of two, their masks alone.
  auto load_raw = [&](const BlockParam *P, int col) {
    if constexpr (NB == 2) {
      vmask = valid_samples(P[0]);
      vmask1 = valid_samples(P[1]);
      live = P[0].state != 0 || P[1].state != 0;
    } else {
      load_column(P[0], col);
    }
  };
  // The words of a thread's 16 samples of the block P that hold the field at bit
  // `off` of each time sample, in w, all on their way before the first is used; of
  // samples not in vm 0.  A field starts at a multiple of its bits, a power of
  // two, so it lies in one word.  Frames and their payloads are whole words, so a
  // word ends within the frame and sample t's field starts at bit (start + NT t
  // ts_bits) mod 32 in whichever frame it lies.  Returns that start.
  auto load_words = [&](const BlockParam &P, int off, unsigned int vm, uint32_t (&w)[16]) {
    const int smp0 = P.nearestsample + jb;
    int q = smp0 / fsamp, r = smp0 - q * fsamp;
    const uint8_t *fr = data + (long long)q * fbytes + 32;
    const int start = (r * D.ts_bits + off) & 31;
#pragma unroll
    for (int t = 0; t < 16; t++) {
      w[t] = load_if(fr + 4 * ((r * D.ts_bits + off) >> 5), (vm >> t) & 1u);
      r += NT;
#pragma unroll 1
      while (r >= fsamp) {
        r -= fsamp;
        fr += fbytes;
      }
    }
    return start;
  };
  // Builds the rotator tables of pair p of the unit P into buf.
  auto build_tables = [&](const BlockParam *P, int p, float2 *buf) {
#pragma unroll
    for (int k = 0; k < SETS; k++) {
      const int bd = NB == 2 ? p : min(2 * p + k, J.nbands - 1);
      put_entries<C>(J, st, st.band_localfreq[bd], st.band_polb[bd], j, P[NB == 2 ? k : 0], D.scale, s_cf, buf + k * T);
    }
  };

  const int b0 = blockIdx.x * G * blocks_per_group + g;
  fetch_param(b0, pbuf);
  fetch_param(b0 + G, pbuf + NB);
  cp_async_wait_all();
  __syncthreads();
  int tb = 0;
  bool staged = false;     // raw and tables hold the block the loop is at
#pragma unroll 1
  for (int it = 0; it < blocks_per_group; it++) {
    const int u = b0 + it * G, bi = u * NB;   // the group's unit and its first block
    if (blockIdx.x * G * blocks_per_group + it * G >= nunit) break;   // no group of the CTA has a unit left
    const BlockParam *const P = pbuf + (it & 1) * NB, *const Pn = pbuf + ((it + 1) & 1) * NB;   // this unit, the group's next one
    if (!staged) {
      load_raw(P, 0);
      build_tables(P, 0, tabs + tb * SETS * T);
    }
    staged = false;
    // blocks that are not processed: zero spectra (all blocks of a warp, where it holds several groups)
    if (NT <= 32 ? !__any_sync(0xffffffffu, live) : !live) {
      for (int b = bi; b < min(nblk, bi + NB); b++)
        for (int bd = 0; bd < J.nbands; bd++) {
          float2 *row = spec + (((size_t)st.freq_index[st.band_localfreq[bd]] * nblk + b) * J.ninputs + st.band_input[bd]) * N;
          for (int c = j; c < N; c += NT) row[c] = make_float2(0.f, 0.f);
        }
      sync_group<NT, CTA>(g);   // all have read this unit's parameters
      fetch_param(u + 2 * G, pbuf + (it & 1) * NB);
      cp_async_wait_all();
      sync_group<NT, CTA>(g);
      continue;
    }
    const bool more = it < blocks_per_group - 1;
#pragma unroll 1
    for (int p = 0; p < D.nfields; p++) {
      // A pair's second band is always there, but has1 stays a condition: without
      // it the compiler runs the two bands' corrections and stores into one another
      // (complex pairs of two frequencies, 16 stations, 1024 points: F-step
      // 0.90 -> 0.96 ms).
      const int bd0 = NB == 2 ? p : 2 * p, bd1 = NB == 2 ? p : min(2 * p + 1, J.nbands - 1);
      const bool has1 = NB == 2 ? bi + 1 < nblk : 2 * p + 1 < J.nbands;
      const int lf0 = st.band_localfreq[bd0], lf1 = SAME || NB == 2 ? lf0 : st.band_localfreq[bd1];
      const float2 *tab0 = tabs + tb * SETS * T, *tab1 = SAME ? tab0 : tab0 + T;
      sync_group<NT, CTA>(g);   // tables written; the previous pair's exchange buffer read
      unsigned int vm0 = vmask, vm1 = NB == 2 ? vmask1 : vmask;
      if (NB == 1 && S.bandmask && bi < nblk && P[0].state != 0) {   // EDV4 masks blank frames per band
        const unsigned long long *bm = S.bandmask + ((size_t)s * nblk + bi) * J.nbands;
        const unsigned long long m0 = bm[bd0], m1 = bm[bd1];
        if (m0 | m1) {
          const int smp0 = P[0].nearestsample + jb;
          int q = smp0 / fsamp, r = smp0 - q * fsamp;
          q -= P[0].fr0;
#pragma unroll 1
          for (int t = 0; t < 16; t++) {
            vm0 &= ~((unsigned int)((m0 >> min(q, 63)) & 1ull) << t);
            vm1 &= ~((unsigned int)((m1 >> min(q, 63)) & 1ull) << t);
            r += NT;
            while (r >= fsamp) {
              r -= fsamp;
              q++;
            }
          }
        }
      }
      if (NB == 2 && S.bandmask) {
#pragma unroll 1
        for (int k = 0; k < NB; k++) {
          const BlockParam &B = P[k];
          if (bi + k >= nblk || B.state == 0) continue;
          const unsigned long long m = S.bandmask[((size_t)s * nblk + bi + k) * J.nbands + p];
          const int smp0 = B.nearestsample + jb;
          int q = smp0 / fsamp, r = smp0 - q * fsamp;
          q -= B.fr0;
#pragma unroll 1
          for (int t = 0; m && t < 16; t++) {
            const unsigned int off = (unsigned int)((m >> min(q, 63)) & 1ull) << t;
            if (k) vm1 &= ~off;
            else vm0 &= ~off;
            r += NT;
            while (r >= fsamp) {
              r -= fsamp;
              q++;
            }
          }
        }
      }
      V v[16];
      float2 psr = dup(0.f), psi = dup(0.f);   // phase-cal: sums of this thread's valid samples
      const int sh = rsh + (p % D.ppc) * D.width;
      {
        // decode and fringe-rotate: x[n] sub[n mod S] step[n / S]; S divides NT,
        // so the sub entry is the same for all 16 samples of the thread
        const float2 rsk0 = tab0[jb & (SD - 1)], rsk1 = SAME ? rsk0 : tab1[jb & (SD - 1)];
        const float4 *rp0 = reinterpret_cast<const float4 *>(tab0 + SD + (jb >> LGS) * 16);
        const float4 *rp1 = reinterpret_cast<const float4 *>(tab1 + SD + (jb >> LGS) * 16);
        auto step = [](const float4 *q, int t) {
          const float4 w = q[t / 2];
          return t & 1 ? make_float2(w.z, w.w) : make_float2(w.x, w.y);
        };
        auto rotate = [&](int t, float2 x, float2 y) {
          if (PC) {
            if ((vm0 >> t) & 1u) { psr.x += x.x; psi.x += y.x; }
            if ((vm1 >> t) & 1u) { psr.y += x.y; psi.y += y.y; }
          }
          const float2 w0 = cmul(rsk0, step(rp0, t));
          const float2 w1 = SAME ? w0 : cmul(rsk1, step(rp1, t));
          if (CPLX) {
            v[t].re = make_float2(w0.x * x.x - w0.y * y.x, w1.x * x.y - w1.y * y.y);
            v[t].im = make_float2(w0.x * y.x + w0.y * x.x, w1.x * y.y + w1.y * x.y);
          } else {
            v[t].re = make_float2(w0.x * x.x, w1.x * x.y);
            v[t].im = make_float2(w0.y * x.x, w1.y * x.y);
          }
        };
        if constexpr (NB == 2) {
          const int nb = J.nbits;
          uint32_t wa[16], wb[16];
          const int s0 = load_words(P[0], p * D.width, vm0, wa), s1 = load_words(P[1], p * D.width, vm1, wb);
#pragma unroll
          for (int t = 0; t < 16; t++) {
            wa[t] >>= (s0 + t * NT * D.ts_bits) & 31;
            wb[t] >>= (s1 + t * NT * D.ts_bits) & 31;
          }
          if (D.kind == 1) {
            const float2 bias = dup(-(float)(8388608 + kCodeOffset));   // as below
#pragma unroll
            for (int t = 0; t < 16; t++) {
              auto part = [&](unsigned int k) {
                return r16::add2(make_float2(__uint_as_float(__byte_perm(wa[t], 0x4B000000u, 0x7650u + k)),
                                             __uint_as_float(__byte_perm(wb[t], 0x4B000000u, 0x7650u + k))), bias);
              };
              rotate(t, part(0), CPLX ? part(1) : dup(0.f));
            }
          } else {
            const uint32_t m = (1u << nb) - 1u;
#pragma unroll
            for (int t = 0; t < 16; t++)
              rotate(t, make_float2(s_lut[wa[t] & m], s_lut[wb[t] & m]),
                     CPLX ? make_float2(s_lut[(wa[t] >> nb) & m], s_lut[(wb[t] >> nb) & m]) : dup(0.f));
          }
        } else if (!fast) {
          // any layout: the fields' own bytes, read here; time samples narrower
          // than a byte start at a bit
          const int smp0 = P[0].nearestsample + jb;
          int q = smp0 / fsamp, r = smp0 - q * fsamp;
          const uint8_t *fr = data + (long long)q * fbytes + 32;
          const int nb = J.nbits, off = D.width * p, nbit = min(D.width, D.ts_bits - off);
          const uint32_t m = (1u << nb) - 1u;
          auto level = [&](uint32_t c) { return D.kind == 1 ? (float)(int)(c & m) - (float)kCodeOffset : s_lut[c & m]; };
#pragma unroll
          for (int t = 0; t < 16; t++) {
            uint32_t f = 0;
            if (((vm0 | vm1) >> t) & 1u) {
              const long long bit = (long long)r * D.ts_bits + off;
              const uint8_t *b = fr + (bit >> 3);
#pragma unroll 1
              for (int k = 0; k == 0 || 8 * k < nbit; k++) f |= (uint32_t)__ldg(b + k) << (8 * k);
              f >>= (int)(bit & 7);
            }
            if (CPLX) rotate(t, make_float2(level(f), level(f >> (2 * nb))), make_float2(level(f >> nb), level(f >> (3 * nb))));
            else rotate(t, make_float2(level(f), level(f >> nb)), dup(0.f));
            r += NT;
#pragma unroll 1
            while (r >= fsamp) {
              r -= fsamp;
              fr += fbytes;
            }
          }
        } else if (D.kind == 0) {
          const uint32_t m = (1u << D.width) - 1u;
#pragma unroll
          for (int t = 0; t < 16; t++) rotate(t, s_pl[(raw[t] >> sh) & m], dup(0.f));
        } else if (D.kind == 1) {
          // code c as the float 2^23 + c (byte placed under the exponent 0x4B)
          const float2 bias = dup(-(float)(8388608 + kCodeOffset));
          const unsigned int s0 = 0x7650u + (unsigned int)(sh >> 3);
#pragma unroll
          for (int t = 0; t < 16; t++) {
            auto byte = [&](unsigned int k) { return __uint_as_float(__byte_perm(raw[t], 0x4B000000u, s0 + k)); };
            if (CPLX) {
              const float2 x = r16::add2(make_float2(byte(0), byte(2)), bias);
              const float2 y = r16::add2(make_float2(byte(1), byte(3)), bias);
              rotate(t, x, y);
            } else {
              rotate(t, r16::add2(make_float2(byte(0), byte(1)), bias), dup(0.f));
            }
          }
        } else {
          const uint32_t m = (1u << J.nbits) - 1u;
          const int nb = J.nbits;
#pragma unroll
          for (int t = 0; t < 16; t++) {
            const uint32_t f = raw[t] >> sh;
            if (CPLX)
              rotate(t, make_float2(s_lut[f & m], s_lut[(f >> (2 * nb)) & m]),
                     make_float2(s_lut[(f >> nb) & m], s_lut[(f >> (3 * nb)) & m]));
            else
              rotate(t, make_float2(s_lut[f & m], s_lut[(f >> nb) & m]), dup(0.f));
          }
        }
        if ((vm0 & vm1) != 0xFFFFu) {
#pragma unroll
          for (int t = 0; t < 16; t++) {
            if (!((vm0 >> t) & 1u)) v[t].re.x = v[t].im.x = 0.f;
            if (!((vm1 >> t) & 1u)) v[t].re.y = v[t].im.y = 0.f;
          }
        }
      }
      if (PC) xb[pc_slot<C>(jb)] = make_float4(psr.x, psr.y, psi.x, psi.y);
      // the next column, or the next block's first one, while the transform runs
      const bool last_pair = p == D.nfields - 1;
      if (last_pair ? more : (p + 1) % D.ppc == 0) load_raw(last_pair ? Pn : P, last_pair ? 0 : (p + 1) / D.ppc);
      const int lsb0 = st.lsb[lf0], lsb1 = SAME ? lsb0 : st.lsb[lf1];
      const float2 sg = make_float2(lsb0 ? -1.f : 1.f, lsb1 ? -1.f : 1.f);   // real data: which half of the bins

      // phase-cal: bin of thread j < nbins, which collects threads j, j + nbins,
      // ... in that order; one thread per bin and block, blocks ordered by the
      // group's barriers, so the sums do not depend on timing
      int pcbin = -1, pcm0 = NT, pcm1 = NT;   // two blocks: bin j, which collects threads pcm0 (pcm1), + nbins, ...
      if (PC && pcout && j < pcn) {
        const unsigned long long n = (unsigned long long)pcn;
        if constexpr (NB == 2) {
          auto first = [&](const BlockParam &B) {
            return (int)(((unsigned long long)j + n - (pcs0 + (unsigned long long)B.nearestsample) % n) % n);
          };
          if (P[0].state != 0) pcm0 = first(P[0]);
          if (P[1].state != 0) pcm1 = first(P[1]);
          if (pcm0 < NT || pcm1 < NT) pcbin = j;
        } else if (P[0].state != 0) {
          pcbin = (int)((pcs0 + (unsigned long long)P[0].nearestsample + (unsigned long long)j) % n);
        }
      }
      auto pcal = [&]() {
        if (PC && pcbin >= 0) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
          float2 *o = pcout + (size_t)bd0 * pf.maxbins + pcbin;
          if constexpr (NB == 2) {
            for (int m = pcm0; m < NT; m += pcn) {
              const float4 q = xb[pc_slot<C>(m)];
              a.x += q.x;
              a.z += q.z;
            }
            for (int m = pcm1; m < NT; m += pcn) {
              const float4 q = xb[pc_slot<C>(m)];
              a.x += q.y;
              a.z += q.w;
            }
          } else {
            for (int m = j; m < NT; m += pcn) {
              const float4 q = xb[pc_slot<C>(m)];
              a.x += q.x;
              a.y += q.y;
              a.z += q.z;
              a.w += q.w;
            }
          }
          atomicAdd(&o->x, a.x * D.scale);
          if (CPLX) atomicAdd(&o->y, a.z * D.scale);
          if (NB == 1) {
            o += pf.maxbins;
            atomicAdd(&o->x, a.y * D.scale);
            if (CPLX) atomicAdd(&o->y, a.w * D.scale);
          }
        }
      };
      // passes: stride 1, then 16 and 256, then the final radix; an exchange between
      dft16<false>(v, sg);
      store16(v, jj, 1, xh);
      sync_half();
      if (PC && !C::SPLIT) pcal();
      load16<C::FS>(v, jj, xh);
      if constexpr (C::L == 1) {
        final_pass<F, C::R0, HALF, !CPLX>(v, j, fin, sg);
      } else {
        pass16<1, HALF && C::L == 2 && C::R0 == 1, !CPLX>(v, jj, twA, twB, sg);
        if constexpr (C::L == 3) {
          sync_half();
          store16(v, jj, 16, xh);
          sync_half();
          load16<C::FS>(v, jj, xh);
          pass16<2, HALF && C::R0 == 1, !CPLX>(v, jj, twA, twB, sg);
        }
        if constexpr (C::SPLIT) {
          // register t holds bin k = jj + NTS t of the half's transform, E or O:
          // X[k] = E[k] + W_F^k O[k], X[k + F / 2] = E[k] - W_F^k O[k].  The
          // even half takes t < 8, the odd half t >= 8: each passes the other
          // eight bins on.
          sync_half();
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const V o = h ? v[i] : v[i + 8];
            xh[r16::pad(jj + C::NTS * i)] = make_float4(o.re.x, o.re.y, o.im.x, o.im.y);
          }
          sync_group<NT, CTA>(g);
          if (PC) pcal();
          const float4 *xo = xb + (1 - h) * (C::FS + C::FS / 16);
          const float2 *w = fin + jj + 8 * C::NTS * h;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const float4 q = xo[r16::pad(jj + C::NTS * i)];
            const V got{make_float2(q.x, q.y), make_float2(q.z, q.w)};
            const V e = h ? got : v[i], o = vmul<!CPLX>(h ? v[i + 8] : got, w[C::NTS * i].x, w[C::NTS * i].y);
            if (HALF) {
              v[i] = vaddsgn(e, o, sg);
            } else {
              v[i] = vadd(e, o);
              v[i + 8] = vsub(e, o);
            }
          }
        } else if constexpr (C::R0 > 1) {
          sync_group<NT, CTA>(g);
          store16(v, j, r16::pow16(C::L - 1), xb);
          sync_group<NT, CTA>(g);
          load16<F>(v, j, xb);
          final_pass<F, C::R0, HALF, !CPLX>(v, j, fin, sg);
        }
      }
      // register t holds one of the kept bins: fractional-sample correction
      // sub[c mod S] step[c / S], store
      if (bi < nblk) {
        // first channel of register 0, and the constant step to register t's
        const int c0 = C::SPLIT ? jj + 8 * C::NTS * h : j;
        auto hop = [](int t) { return C::SPLIT ? C::NTS * (t < 8 ? t : t + 8) : NT * t; };
        auto pick = [&](int t, int lane) {
          return lane ? make_float2(v[t].re.y, v[t].im.y) : make_float2(v[t].re.x, v[t].im.x);
        };
        // the thread's steps: consecutive, from register 0's channel on (a split
        // group's upper eight registers are 16 steps on)
        const int s0 = (jj >> LGS) * (N / C::NTS) + (C::SPLIT ? 8 * h : 0);
        // register t's channel and whether its value is conjugated (complex lower sideband)
        auto channel = [&](int t, int lsb, bool &conj) {
          const int bin = c0 + hop(t);
          conj = CPLX && lsb && bin != 0;
          return conj ? F - bin : bin;
        };
        // its correction from a band's tables
        auto corr = [&](const float2 *tab, int lsb, int t) {
          const float2 *fs = tab + SD + C::NFR, *fp = fs + SD;
          if (CPLX && lsb) {
            bool conj;
            const int c = channel(t, lsb, conj);
            return cmul(fs[(-jj) & (SD - 1)], fp[step_pos<C::NTS, SD>(c >> LGS, N / C::NTS)]);
          }
          const float4 q = reinterpret_cast<const float4 *>(fp + s0)[(C::SPLIT && t >= 8 ? t + 8 : t) / 2];
          return cmul(fs[jj & (SD - 1)], t & 1 ? make_float2(q.z, q.w) : make_float2(q.x, q.y));
        };
        auto value = [&](int t, int lane, bool conj) {
          float2 val = pick(t, lane);
          if (conj) val.y = -val.y;
          return val;
        };
        if (SAME) {
          // both bands by the same correction
          const size_t base = ((size_t)st.freq_index[lf0] * nblk + bi) * J.ninputs;
          float2 *row0 = spec + (base + st.band_input[bd0]) * N;
          float2 *row1 = spec + (base + st.band_input[bd1]) * N;
          auto both = [&](int lsb, bool paired) {
#pragma unroll
            for (int t = 0; t < NOUT; t++) {
              bool conj;
              const int c = channel(t, lsb, conj);
              const float2 w = corr(tab0, lsb, t);
              const float2 x = cmul(value(t, 0, conj), w), y = cmul(value(t, 1, conj), w);
              if (paired) {
                reinterpret_cast<float4 *>(row0)[c] = make_float4(x.x, x.y, y.x, y.y);
              } else {
                row0[c] = x;
                if (has1) row1[c] = y;
              }
            }
          };
          if (CPLX && lsb0) J.paired ? both(1, true) : both(1, false);
          else J.paired ? both(0, true) : both(0, false);
        } else {
          auto one = [&](int lane, const float2 *tab, int bd, int lf, int lsb) {
            const int b = NB == 2 ? bi + lane : bi;
            float2 *row = spec + (((size_t)st.freq_index[lf] * nblk + b) * J.ninputs + st.band_input[bd]) * N;
#pragma unroll
            for (int t = 0; t < NOUT; t++) {
              bool conj;
              const int c = channel(t, lsb, conj);
              row[c] = cmul(value(t, lane, conj), corr(tab, lsb, t));
            }
          };
          auto emit = [&](int lane, const float2 *tab, int bd, int lf, int lsb) {
            if (CPLX && lsb) one(lane, tab, bd, lf, 1);
            else one(lane, tab, bd, lf, 0);
          };
          emit(0, tab0, bd0, lf0, lsb0);
          if (has1) emit(1, tab1, bd1, lf1, lsb1);
        }
      }
      if constexpr (C::TBUF == 1) sync_group<NT, CTA>(g);   // the tables are rewritten in place
      if (!last_pair || more) {
        // every thread has read this unit's parameters before the exchanges'
        // synchronisation: the buffer takes those of the unit after the next
        if (last_pair) fetch_param(u + 2 * G, pbuf + (it & 1) * NB);
        tb ^= C::TBUF - 1;
        build_tables(last_pair ? Pn : P, last_pair ? 0 : p + 1, tabs + tb * SETS * T);
        if (last_pair) cp_async_wait_all();
      }
    }
    staged = more;
  }
}

#define GX_PAIR_ARGS                                                                                               \
  const DevJob &J, const DevStation *stations, const SubintArrays &S, int nblk, int items, const PairDecode &D,   \
      const BlockParam *bp, float2 *spec, const PcalFuse &pf, cudaStream_t st

// Launches the kernel of a transform length for one data type; ONE: one band and
// two blocks at a time, else the pairs.
template <int CPLX, bool PC, bool ONE>
cudaError_t launch(GX_PAIR_ARGS)
{
  const bool same = J.pair_same != 0;
  auto go = [&](auto kernel, int groups, int cta, size_t sm) -> cudaError_t {
    cudaError_t e = smem_opt_in((const void *)kernel, sm);
    if (e != cudaSuccess) return e;
    const int nunit = ONE ? (nblk + 1) / 2 : nblk;
    const dim3 grid((nunit + items * groups - 1) / (items * groups), J.nstations);
    kernel<<<grid, cta, sm, st>>>(J, stations, S, bp, nblk, items, D, spec, pf);
    return cudaGetLastError();
  };
#define GX_PAIR_FORM(FLV, LANES) \
  go(fstep_pair_kernel<FLV, CPLX, LANES, PC>, Cfg<FLV, CPLX>::G, Cfg<FLV, CPLX>::CTA, smem_bytes<FLV, CPLX, LANES>())
#define GX_PAIR_CASE(FLV)                                                                                  \
  case FLV:                                                                                                \
    if constexpr (ONE) return GX_PAIR_FORM(FLV, kTwoBlocks);                                               \
    else return same ? GX_PAIR_FORM(FLV, kSameBands) : GX_PAIR_FORM(FLV, kTwoBands);
  switch (J.fftlen) {
    GX_PAIR_CASE(128)
    GX_PAIR_CASE(256)
    GX_PAIR_CASE(512)
    GX_PAIR_CASE(1024)
    GX_PAIR_CASE(2048)
    GX_PAIR_CASE(4096)
    GX_PAIR_CASE(8192)
  }
#undef GX_PAIR_CASE
#undef GX_PAIR_FORM
  return cudaErrorNotSupported;
}

// one translation unit each: the kernels of a data type, and of one band at a
// time, without and with phase-cal
cudaError_t launch_real(GX_PAIR_ARGS);
cudaError_t launch_cplx(GX_PAIR_ARGS);
cudaError_t launch_real_pc(GX_PAIR_ARGS);
cudaError_t launch_cplx_pc(GX_PAIR_ARGS);
cudaError_t launch_one(GX_PAIR_ARGS);
cudaError_t launch_one_pc(GX_PAIR_ARGS);

}  // namespace pr
}  // namespace gx
