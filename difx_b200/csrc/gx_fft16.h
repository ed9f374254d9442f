// Register-resident forward FFT of F points spread over NT = F / 16 threads
// (16 points per thread), the building block of the long-transform F-step.
//
// Stockham formulation: every pass reads the 16 points x[j + NT t] of thread j
// (t = 0..15).  A radix-16 pass of stride Ns twiddles them by W_{16 Ns}^{(j mod Ns) r},
// transforms them in registers (16 = 4 x 4) and writes them to
// out[(j - j mod Ns) * 16 + j mod Ns + Ns r] in shared memory, padded by one
// element every 16 so that the strided stores and loads spread over the banks.
// With F = 16^L * R0 (R0 in {1, 2, 4, 8}) the last radix-16 pass (R0 = 1) or a
// final radix-R0 pass (16 / R0 transforms per thread, done in registers) leaves
// X[j + NT t] in register t of thread j: no exchange after the last pass.
//
// Everything here is __host__ __device__ so that the index arithmetic can be
// exercised on the CPU.
#pragma once
#include <cuda_runtime.h>

namespace gx {
namespace r16 {

__host__ __device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ float2 mul(float2 a, float2 b)
{
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// shared-memory position of element i: one pad element per 16
__host__ __device__ __forceinline__ int pad(int i) { return i + (i >> 4); }

// Paired FP32 add and subtract (one f32x2 instruction on sm_100, same
// rounding as the two scalar operations); plain float2 arithmetic on the host.
__host__ __device__ __forceinline__ float2 add2(float2 a, float2 b)
{
#ifdef __CUDA_ARCH__
  return __fadd2_rn(a, b);
#else
  return add(a, b);
#endif
}
__host__ __device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
#ifdef __CUDA_ARCH__
  float2 r;
  asm("{\n\t.reg .b64 pa, pb, pd;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
      "sub.rn.f32x2 pd, pa, pb;\n\tmov.b64 {%0, %1}, pd;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
#else
  return sub(a, b);
#endif
}

__host__ __device__ constexpr int log16_floor(int f) { return f >= 65536 ? 4 : (f >= 4096 ? 3 : (f >= 256 ? 2 : (f >= 16 ? 1 : 0))); }
__host__ __device__ constexpr int pow16(int l) { return l == 0 ? 1 : 16 * pow16(l - 1); }

// Twiddle table of an F-point transform as the device holds it: W_F^m for m
// in [0, F); then one section per radix-16 pass of stride Ns = 16^p
// (p = 1 .. L - 1), entry (r - 1) Ns + m = W_F^(r m F / (16 Ns)); then, for a
// final radix R0 > 1, entry (r - 1) (F / R0) + g = W_F^(g r).  Each row holds
// consecutive m (or g), so the loads of one r by a warp are contiguous.
__host__ __device__ constexpr int tw_pass_offset(int F, int p)
{
  int o = F;
  for (int q = 1; q < p; q++) o += 15 * pow16(q);
  return o;
}
__host__ __device__ constexpr int tw_final_offset(int F) { return tw_pass_offset(F, log16_floor(F)); }
__host__ __device__ constexpr int tw_table_size(int F)
{
  return tw_final_offset(F) + (F / pow16(log16_floor(F)) > 1 ? (F / pow16(log16_floor(F)) - 1) * pow16(log16_floor(F)) : 0);
}

}  // namespace r16
}  // namespace gx
