// X-step (plain FP32 form): Hermitian cross-multiply-accumulate of the
// spectra of every input (station x band) of a frequency, per channel,
// summed over FFT blocks -- the work of Core::processdata's XMAC loop
// (mpifxcorr/src/core.cpp:884-968, vectorAddProduct_cf32 ->
// genericAddProduct_32fc, architecture.h.in:575-580) and of the station
// autocorrelations (mode.cpp:1270-1285, 1333-1352), which are the diagonal
// and same-station entries of the same Hermitian product.
//
// Work decomposition: the NI x NI input matrix of a frequency is split into
// ST x ST super-tiles; only super-tiles on or above the diagonal are
// computed, and on the diagonal only the register tiles that reach the upper
// triangle.  A CTA owns one super-tile for CT channels and a slice of the
// blocks; each thread owns an 8 x TB register tile of accumulators for one
// channel.  Spectra rows of the super-tile are staged in shared memory.
//
// Accumulators: acc[ks][freq][stpair][ST][ST][N] (float2), summed over the
// chunk passes of a subint; finalise_kernel maps them to the Core result
// layout (configuration.cpp:2348-2630) and sums the K-split slices.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include "gx_dev.h"
#include "gx_xstep.h"
#include "gx_mbar.cuh"
#include "gx_fcommon.cuh"

namespace gx {

// Register tiles of a super-tile pair: kTA rows by TB columns.  On the diagonal
// only those that reach the upper triangle (in whole groups of kTA rows).
constexpr int kTA = 8;
template <int TB, int ST, bool DIAG>
__host__ __device__ constexpr int xmac_tiles()
{
  int n = 0;
  for (int i = 0; i < ST / kTA; i++) n += DIAG ? (ST - kTA * i) / TB : ST / TB;
  return n;
}
// Consumer warps of a CTA: two tiles by 16 channels each.
template <int TB, int ST, int CT, bool DIAG>
__host__ __device__ constexpr int xmac_warps() { return xmac_tiles<TB, ST, DIAG>() / 2 * (CT / 16); }

// Blocks that a product is summed over in one register, at most.
__host__ __device__ constexpr int xmac_run(bool two) { return two ? 96 : 256; }

// One CTA: super-tile pair blockIdx.x (DIAG: the pairs on the diagonal, else
// those above it, row-major) of frequency f for CT channels from c0 =
// blockIdx.y CT, over the blocks of K-split slice ks.  Stages -- KB blocks x ST
// rows x CT channels of the I and (off the diagonal) J rows, one TMA tile per
// operand -- go round an NSTAGE ring: the warp that is last to finish with a
// stage loads the next one into its place, so there is neither a producer warp
// (a 21st warp would cost every thread of a 20-warp CTA 16 registers) nor a
// barrier between the stages.  accumulate 0: the sums are stored, not added to
// what acc holds.  Every wait is bounded (kWaitLimitNs): on expiry the CTA
// records a status in *err (when given), drains the copies it issued and adds
// nothing more.
//
// What bounds it: the FMA pipe.  Only the register tiles that reach the upper
// triangle have threads (32 inputs: 20 tiles of 8 x 4; a thread for each 8 x 8
// tile of the square left 6 of 16 idle), and 8 x 4 tiles let 20 warps an SM hide
// the shared-memory latency.  64 stations, 4096 channels, 125 blocks: 5.41 ->
// 2.77 ms, 26 of the 36 T FMA lanes a second that 128 a clock are (16 stations,
// 6250 blocks: 2.81 -> 1.18 ms, 28 of them).
// The sums of a product stay short: after a run of blocks in one register, TWO
// register levels (where the shape leaves the registers) or the accumulators in
// memory take them over, so the FP32 error does not grow with the pass.  A slice
// is cut into equal runs of at most xmac_run(TWO) blocks: runs of the longest
// length and a rest cost the same and err more (16 stations, 5000 blocks in slices
// of 320: 4.0e-7 of the 64-bit values in runs of 256 and 64, 3.6e-7 in two of 160).
template <int TB, int ST, int CT, int KB, int NSTAGE, bool DIAG, int MINB, bool TWO>
__global__ void __launch_bounds__(xmac_warps<TB, ST, CT, DIAG>() * 32, MINB)
xmac_fp32_kernel(const __grid_constant__ CUtensorMap spec_map, int nblk, int N, int nsuper, int ks_count,
                 int kper, int run_stages, float2 *__restrict__ acc, int accumulate, int *__restrict__ err)
{
  constexpr int NCW = xmac_warps<TB, ST, CT, DIAG>();
  constexpr int NTILE = xmac_tiles<TB, ST, DIAG>();
  constexpr int STAGE = KB * ST * CT;   // float2 per stage per operand
  static_assert(NTILE % 2 == 0 && CT % 16 == 0 && ST % kTA == 0 && kTA % TB == 0, "a warp takes two tiles by 16 channels");
  extern __shared__ __align__(128) float2 xsm[];
  float2 *sI = xsm;                     // [NSTAGE][KB][ST][CT]
  float2 *sJ = DIAG ? sI : xsm + NSTAGE * STAGE;
  uint64_t *full = reinterpret_cast<uint64_t *>(xsm + (DIAG ? 1 : 2) * NSTAGE * STAGE);
  int *s_done = reinterpret_cast<int *>(full + NSTAGE);   // warps done with each stage's current contents
  volatile int *s_issued = s_done + NSTAGE;
  volatile int *s_abort = s_done + NSTAGE + 1;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c0 = blockIdx.y * CT;
  const int f = blockIdx.z / ks_count;
  const int ks = blockIdx.z % ks_count;
  int SI, SJ;
  if (DIAG) {
    SI = SJ = blockIdx.x;
  } else {
    int rem = blockIdx.x;
    SI = 0;
    while (rem >= nsuper - 1 - SI) { rem -= nsuper - 1 - SI; SI++; }
    SJ = SI + 1 + rem;
  }
  const int stp = SI * nsuper - SI * (SI - 1) / 2 + (SJ - SI);   // place among all upper pairs
  const int I0 = SI * ST, J0 = SJ * ST;

  // slices start on stage boundaries (kper is a multiple of KB); the last
  // stage may reach past nblk, where the copies read zeros
  const int kb0 = ks * kper, kb1 = min(nblk, kb0 + kper);
  const int nstages = (kb1 > kb0) ? (kb1 - kb0 + KB - 1) / KB : 0;

  auto load_stage = [&](int st) {   // one thread
    const int b = st % NSTAGE, k = kb0 + st * KB;
    const uint32_t bar = smem_u32(full + b);
    mbar_expect_tx(bar, (DIAG ? 1u : 2u) * (uint32_t)(STAGE * sizeof(float2)));
    tma_load_4d(smem_u32(sI + b * STAGE), &spec_map, 2 * c0, I0, k, f, bar);
    if (!DIAG) tma_load_4d(smem_u32(sJ + b * STAGE), &spec_map, 2 * c0, J0, k, f, bar);
    *s_issued = st + 1;   // stages are issued in order
  };
  if (tid == 0) {
    for (int i = 0; i < NSTAGE; i++) {
      mbar_init(smem_u32(full + i), 1);
      s_done[i] = 0;
    }
    *s_abort = 0;
    *s_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async_smem();
    for (int i = 0; i < NSTAGE && i < nstages; i++) load_stage(i);
  }
  __syncthreads();
  auto abort_with = [&](int code) {
    *s_abort = 1;
    if (err) atomicExch(err, code);
  };

  // ---- consumers: a kTA x TB register tile of one channel; a warp takes two
  // neighbouring tiles (mostly of the same rows) by 16 channels, so that its
  // row loads are whole 128-byte lines
  const int c = (warp / (NTILE / 2)) * 16 + (lane & 15);
  int ti = 0, tj = 2 * (warp % (NTILE / 2)) + (lane >> 4);
  if (DIAG) {
    while (tj >= (ST - kTA * ti) / TB) { tj -= (ST - kTA * ti) / TB; ti++; }
    tj += kTA / TB * ti;
  } else {
    ti = tj / (ST / TB);
    tj %= ST / TB;
  }
  float2 acc2[kTA][TB];   // (Re, Im) of each product sum, one register pair for the f32x2 FMAs
#pragma unroll
  for (int a = 0; a < kTA; a++)
#pragma unroll
    for (int b = 0; b < TB; b++) acc2[a][b] = make_float2(0.f, 0.f);
  float2 tot[TWO ? kTA : 1][TWO ? TB : 1];   // the finished runs' sums
  if constexpr (TWO) {
#pragma unroll
    for (int a = 0; a < kTA; a++)
#pragma unroll
      for (int b = 0; b < TB; b++) tot[a][b] = make_float2(0.f, 0.f);
  }
  const int nfreqs = gridDim.z / ks_count, npairs = nsuper * (nsuper + 1) / 2;
  float2 *tile = acc + ((((size_t)ks * nfreqs + f) * npairs + stp) * (size_t)ST * ST + (ti * kTA) * ST + tj * TB) * N + c0 + c;
  // adds (or stores) the tile's sums x
  auto put = [&](const float2 (&x)[kTA][TB], bool add) {
    if (c0 + c >= N) return;
    float2 *t = tile;
    asm volatile("" : "+l"(t));   // no addresses formed ahead: they would cost the loop its registers
#pragma unroll
    for (int a = 0; a < kTA; a++, t += (size_t)ST * N) {
      float2 old[TB];   // a row's loads together: one by one, behind the stores, their latency was a tenth of a pass
      if (add) {
#pragma unroll
        for (int b = 0; b < TB; b++) old[b] = t[(size_t)b * N];
      }
#pragma unroll
      for (int b = 0; b < TB; b++) {
        float2 v = x[a][b];
        if (add) v = make_float2(v.x + old[b].x, v.y + old[b].y);
        t[(size_t)b * N] = v;
      }
    }
  };
  bool ok = true, add = accumulate != 0;
  int st = 0;
#pragma unroll 1
  do {
    const int run = min(nstages, st + run_stages);
#pragma unroll 1
    for (; st < run; st++) {
      const int buf = st % NSTAGE;
      const bool good = mbar_wait(smem_u32(full + buf), (uint32_t)(st / NSTAGE) & 1u);
      const float2 *bi_ = sI + buf * STAGE + ti * kTA * CT + c;
      const float2 *bj_ = sJ + buf * STAGE + tj * TB * CT + c;
#pragma unroll 1
      for (int kk = 0; kk < KB; kk++) {
        // xi * conj(xj) as two paired FMAs (one f32x2 instruction each on
        // sm_100): Re += xi.x xj.x then xi.y xj.y; Im += xi.y xj.x then -xi.x xj.y,
        // the same operations in the same order as four scalar FMAs.
        float2 bx[TB], by[TB];
#pragma unroll
        for (int r = 0; r < TB; r++) {
          const float2 xj = bj_[(kk * ST + r) * CT];
          bx[r] = make_float2(xj.x, xj.x);
          by[r] = make_float2(xj.y, xj.y);
        }
#pragma unroll
        for (int a = 0; a < kTA; a++) {
          const float2 xi = bi_[(kk * ST + a) * CT];
          const float2 xs = make_float2(xi.y, -xi.x);
#pragma unroll
          for (int b = 0; b < TB; b++) acc2[a][b] = __ffma2_rn(xi, bx[b], acc2[a][b]);
#pragma unroll
          for (int b = 0; b < TB; b++) acc2[a][b] = __ffma2_rn(xs, by[b], acc2[a][b]);
        }
      }
      if (!stage_end(good)) {
        abort_with(14);
        ok = false;
        break;
      }
      if (lane == 0) {
        // done with the stage: the last warp to be (its acquire follows every
        // other's release, so all reads of the stage precede the copy) refills it
        int before;
        asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(smem_u32(s_done + buf)) : "memory");
        if (before == NCW - 1 && st + NSTAGE < nstages && !*s_abort) {
          s_done[buf] = 0;
          load_stage(st + NSTAGE);
        }
      }
    }
    if (!ok) break;
    if constexpr (TWO) {
#pragma unroll
      for (int a = 0; a < kTA; a++)
#pragma unroll
        for (int b = 0; b < TB; b++) {
          tot[a][b] = make_float2(tot[a][b].x + acc2[a][b].x, tot[a][b].y + acc2[a][b].y);
          acc2[a][b] = make_float2(0.f, 0.f);
        }
    } else {
      put(acc2, add);
      add = true;
#pragma unroll
      for (int a = 0; a < kTA; a++)
#pragma unroll
        for (int b = 0; b < TB; b++) acc2[a][b] = make_float2(0.f, 0.f);
    }
  } while (st < nstages);
  if (*s_abort) ok = false;
  if (__syncthreads_or(!ok)) {
    // drain: the copies this CTA issued land before it exits (bounded)
    if (tid == 0) {
      const int issued = *s_issued;
      for (int b = 0; b < NSTAGE && b < issued; b++) {
        const int ulast = b + ((issued - 1 - b) / NSTAGE) * NSTAGE;
        mbar_wait(smem_u32(full + b), (uint32_t)(ulast / NSTAGE) & 1u);
      }
    }
    __syncthreads();
    return;
  }
  if constexpr (TWO) put(tot, add);
}

// Sum of weights over the blocks of one chunk (Core::processdata baseline
// weights core.cpp:1005-1052; Mode autocorrelation weights mode.cpp:1277-1284).
// Weight sums over a pass of blocks: item i < nstations sums station row i;
// item nstations + k sums the products of rows pairs[k] (or row pairs[k].x
// alone when pairs[k].y < 0).
constexpr int kWeightThreads = 1024;
__global__ void __launch_bounds__(kWeightThreads)
weights_kernel(const float *__restrict__ w, int nblk, int nstations, const int2 *__restrict__ pairs, int npairs,
               float *__restrict__ wacc, int accumulate)
{
  __shared__ float red[kWeightThreads / 32];
  const int item = blockIdx.x;  // [0, nstations): station sums; then baseline products
  const int2 pr = item < nstations ? make_int2(item, -1) : pairs[item - nstations];
  const float *x = w + (size_t)pr.x * nblk;
  const float *y = pr.y < 0 ? nullptr : w + (size_t)pr.y * nblk;   // null: one row alone
  float sum = 0.f;
  // several loads in flight: a CTA reads whole rows, and there are few CTAs
#pragma unroll 4
  for (int b = threadIdx.x; b < nblk; b += kWeightThreads) sum += y ? x[b] * y[b] : x[b];
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x < 32) {
    sum = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (threadIdx.x == 0) wacc[item] = accumulate ? wacc[item] + sum : sum;
  }
}

__device__ __forceinline__ void finalise_weight(const WeightEntry *__restrict__ we, int nw, int e,
                                                const float *__restrict__ wacc, float *__restrict__ results_f)
{
  if (e >= nw) return;
  const WeightEntry x = we[e];
  results_f[x.float_index] = x.source >= 0 ? wacc[x.source] : 0.0f;
}

// Result array assembly (Core result layout): one product row by up to 4
// blockDim channels, four a thread; the CTAs after the nprods rows' write the
// weights.  Bound by HBM (accumulators in, results out): several loads a thread
// cover its latency (64 stations, 4096 channels, with nothing cleared first: 0.83 ->
// 0.46 ms).
__global__ void finalise_vis_kernel(const ProdEntry *__restrict__ prods, int nprods, const float2 *__restrict__ acc,
                                    int ks_count, size_t ks_stride, int N, const WeightEntry *__restrict__ we, int nw,
                                    const float *__restrict__ wacc, float2 *__restrict__ results)
{
  if ((int)blockIdx.x >= nprods) {
    if (blockIdx.y == 0)
      finalise_weight(we, nw, (blockIdx.x - nprods) * blockDim.x + threadIdx.x, wacc, reinterpret_cast<float *>(results));
    return;
  }
  const ProdEntry pe = prods[blockIdx.x];
  const int c0 = blockIdx.y * 4 * blockDim.x + threadIdx.x;
  const float2 *a = acc + pe.acc_index + c0;
  float2 *out = results + pe.result_offset + c0;
  // One channel a thread: eight slices' reads in flight instead of four
  // channels' (jobs of few inputs cut a pass into many slices: 16 stations 54 -> 33 us,
  // 4 stations of 128 channels 23 -> 8).  With 4 channels a thread as well, the
  // 64-station 4096-channel job was slower (0.46 -> 0.55 ms): it keeps the form below.
  if (N <= (int)blockDim.x) {
    if (c0 >= N) return;
    // four sums of every fourth slice, then those: with up to 64 slices one sum
    // after the other would err more than the slices themselves (11 stations of
    // 64 channels, 37 slices: 1.3e-7 of the 64-bit values, 1.0e-7 in four)
    float2 p[4];
#pragma unroll
    for (int i = 0; i < 4; i++) p[i] = make_float2(0.f, 0.f);
    int k = 0;
#pragma unroll 2
    for (; k + 4 <= ks_count; k += 4)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float2 v = a[(size_t)(k + i) * ks_stride];
        p[i].x += v.x;
        p[i].y += v.y;
      }
    for (; k < ks_count; k++) {
      const float2 v = a[(size_t)k * ks_stride];
      p[0].x += v.x;
      p[0].y += v.y;
    }
    const float re = (p[0].x + p[1].x) + (p[2].x + p[3].x), im = (p[0].y + p[1].y) + (p[2].y + p[3].y);
    out[0] = make_float2(re, pe.conj ? -im : im);
    return;
  }
  float2 s[4];
#pragma unroll
  for (int i = 0; i < 4; i++)
    s[i] = c0 + i * (int)blockDim.x < N ? a[i * blockDim.x] : make_float2(0.f, 0.f);
#pragma unroll 2
  for (int k = 1; k < ks_count; k++) {
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (c0 + i * (int)blockDim.x < N) {
        const float2 v = a[(size_t)k * ks_stride + i * blockDim.x];
        s[i].x += v.x;
        s[i].y += v.y;
      }
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
    if (c0 + i * (int)blockDim.x < N) out[i * blockDim.x] = make_float2(s[i].x, pe.conj ? -s[i].y : s[i].y);
}

__global__ void finalise_weights_kernel(const WeightEntry *__restrict__ we, int nw, const float *__restrict__ wacc,
                                        float *__restrict__ results_f)
{
  finalise_weight(we, nw, blockIdx.x * blockDim.x + threadIdx.x, wacc, results_f);
}

// ------------------------------------------------------------------ launchers

template <int TB, int ST, int CT, int KB, int NSTAGE, bool DIAG, int MINB, bool TWO>
static cudaError_t launch_t(const float2 *spec, int nblk, int rows, int NI, int N, int nfreqs, int ks, float2 *acc,
                            int accumulate, int *err, cudaStream_t st)
{
  const int nsuper = (NI + ST - 1) / ST;
  const int npairs = DIAG ? nsuper : nsuper * (nsuper - 1) / 2;
  if (npairs == 0) return cudaSuccess;
  const size_t sm = sizeof(float2) * (DIAG ? 1 : 2) * NSTAGE * KB * ST * CT + NSTAGE * (sizeof(uint64_t) + sizeof(int)) + 16;
  // spec[freq][block][row][channel] float2 as a 4-D FP32 tensor: {2N floats,
  // rows in use (the others of the NI are not read), nblk blocks, nfreqs}; one
  // box = KB blocks x ST rows x CT channels
  CUtensorMap map;
  const cuuint64_t dims[4] = {(cuuint64_t)(2 * N), (cuuint64_t)rows, (cuuint64_t)nblk, (cuuint64_t)nfreqs};
  const cuuint32_t box[4] = {(cuuint32_t)(2 * CT), (cuuint32_t)ST, (cuuint32_t)KB, 1};
  cudaError_t e = tma_map_f32_4d(&map, spec, dims, box, NI);
  if (e != cudaSuccess) return e;
  auto kernel = xmac_fp32_kernel<TB, ST, CT, KB, NSTAGE, DIAG, MINB, TWO>;
  e = smem_opt_in((const void *)kernel, sm);
  if (e != cudaSuccess) return e;
  // slices of whole stages, on 16-block boundaries for every variant, so that
  // the variants add the same blocks into each slice
  static_assert(16 % KB == 0, "slice boundaries must be whole stages");
  const int kper = ((nblk + ks - 1) / ks + 15) / 16 * 16;
  const int units = kper / 16, runs = (units * 16 + xmac_run(TWO) - 1) / xmac_run(TWO);
  const int run_stages = (units + runs - 1) / runs * (16 / KB);
  // super-tile pairs fastest: the pairs that share a channel group's spectra run together
  dim3 grid(npairs, (N + CT - 1) / CT, nfreqs * ks);
  kernel<<<grid, xmac_warps<TB, ST, CT, DIAG>() * 32, sm, st>>>(map, nblk, N, nsuper, ks, kper, run_stages, acc, accumulate, err);
  return cudaGetLastError();
}

// Channels per CTA: 20 warps of 20 tiles by 32 channels where one super-tile
// holds every input (16 stations, 2-bit, 6250 blocks: X stage 2.81 -> 1.18 ms;
// 16 channels and two CTAs an SM 1.34, 8 x 8 tiles 1.66 before longer passes),
// as on the diagonal of larger ones; 12 warps of 6 tiles by 64 channels for 16
// rows (11 stations: 0.42 ms, two CTAs of 32 channels 0.54, the square of 4 x 4
// tiles 0.66); two warps of two tiles by 32 channels for 8 rows (4 stations, 25000
// blocks: 0.17 ms, 64 channels 0.18, 4 x 4 tiles 0.36).
XmacShape xmac_shape(int NI)
{
  XmacShape s;
  s.T = kTA;
  if (NI <= 8) { s.ST = 8; s.CT = 32; }
  else if (NI <= 16) { s.ST = 16; s.CT = 64; }
  else { s.ST = 32; s.CT = NI <= 32 ? 32 : 16; }
  s.nsuper = (NI + s.ST - 1) / s.ST;
  s.npairs = s.nsuper * (s.nsuper + 1) / 2;
  return s;
}

cudaError_t xmac_fp32_launch(const float2 *spec, int nblk, int rows, int NI, int N, int nfreqs, int ks, float2 *acc,
                             int accumulate, int *err, cudaStream_t st, int variant)
{
  // every variant keeps the super-tile ST of the shape (the accumulator
  // layout); variant 1 takes half (or twice) the channels per CTA
  const XmacShape s = xmac_shape(NI);
#define GX_XMAC(TB, ST, CT, KB, DG, MB) \
  launch_t<TB, ST, CT, KB, 3, DG, MB, (ST < 32)>(spec, nblk, rows, NI, N, nfreqs, ks, acc, accumulate, err, st)
  if (s.ST == 8) return variant == 1 ? GX_XMAC(4, 8, 64, 4, true, 3) : GX_XMAC(4, 8, 32, 8, true, 4);
  if (s.ST == 16) return variant == 1 ? GX_XMAC(4, 16, 32, 8, true, 2) : GX_XMAC(4, 16, 64, 8, true, 1);
  cudaError_t e = variant == 1 ? GX_XMAC(4, 32, 16, 8, true, 2) : GX_XMAC(4, 32, 32, 8, true, 1);
  if (e != cudaSuccess) return e;
  // above the diagonal: 8 x 8 tiles, half the shared-memory reads a product of
  // 8 x 4 (64 stations, 125 blocks: 1.98 against 2.06 ms)
  return variant == 1 ? GX_XMAC(4, 32, 16, 8, false, 1) : GX_XMAC(8, 32, 16, 8, false, 1);
#undef GX_XMAC
}

cudaError_t weights_launch(const float *w, int nblk, int nstations, const int2 *pairs, int npairs, float *wacc,
                           int accumulate, cudaStream_t st)
{
  weights_kernel<<<nstations + npairs, kWeightThreads, 0, st>>>(w, nblk, nstations, pairs, npairs, wacc, accumulate);
  return cudaGetLastError();
}

cudaError_t finalise_launch(const ProdEntry *prods, int nprods, const float2 *acc, int ks, size_t ks_stride, int N,
                            const WeightEntry *we, int nw, const float *wacc, float2 *results, cudaStream_t st)
{
  if (nprods > 0) {
    // few channels: one a thread, so that the rows' CTAs fill the chip
    const int threads = N <= 256 ? std::max(32, (N + 31) / 32 * 32) : 256;
    const dim3 grid(nprods + (nw + threads - 1) / threads, (N + 4 * threads - 1) / (4 * threads));
    finalise_vis_kernel<<<grid, threads, 0, st>>>(prods, nprods, acc, ks, ks_stride, N, we, nw, wacc, results);
  } else if (nw > 0)
    finalise_weights_kernel<<<(nw + 255) / 256, 256, 0, st>>>(we, nw, wacc, reinterpret_cast<float *>(results));
  return cudaGetLastError();
}

// Zoom spectra rows: one thread per channel of one row of one block.
__global__ void zoom_gather_kernel(const ZoomRow *__restrict__ rows, const float2 *__restrict__ spec, int NIm, int Nm,
                                   float2 *__restrict__ specz, int NIz, int Nz, int nblk)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= Nz) return;
  const ZoomRow r = rows[blockIdx.y];
  const int b = blockIdx.z;
  specz[(((size_t)r.zf * nblk + b) * NIz + r.zrow) * Nz + k] = spec[(((size_t)r.mf * nblk + b) * NIm + r.mrow) * Nm + r.off + k];
}

cudaError_t zoom_gather_launch(const ZoomRow *rows, int nrows, const float2 *spec, int NIm, int Nm, float2 *specz,
                               int NIz, int Nz, int nblk, cudaStream_t st)
{
  if (nrows <= 0 || nblk <= 0) return cudaSuccess;
  if (nrows > 65535 || nblk > 65535) return cudaErrorInvalidConfiguration;
  dim3 grid((Nz + 127) / 128, nrows, nblk);
  zoom_gather_kernel<<<grid, 128, 0, st>>>(rows, spec, NIm, Nm, specz, NIz, Nz, nblk);
  return cudaGetLastError();
}

// One interval of a multi-phase-centre subint: each thread one channel of
// one product row.  The rotator of channel c is the reference's two-level
// one: sub[c mod rsl] (band-edge turns included) times step[c / rsl], FP64
// turns, FP32 arguments and sincos, FP32 products in the reference's order.
__global__ void uvshift_kernel(const UvEntry *__restrict__ ents, const float2 *__restrict__ acc, int ks,
                               size_t ks_stride, int N, const double *__restrict__ delays, int npc, int maxpc,
                               const UvFreq *__restrict__ freqs, int rsl, float2 *__restrict__ results)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  const UvEntry e = ents[blockIdx.y];
  float2 v = make_float2(0.f, 0.f);
  for (int k = 0; k < ks; k++) {
    const float2 a = acc[(size_t)k * ks_stride + e.acc_index + c];
    v.x += a.x;
    v.y += a.y;
  }
  if (e.conj) v.y = -v.y;
  if (e.stride == 0) {
    float2 &r = results[e.ro + c];
    r.x += v.x;
    r.y += v.y;
    return;
  }
  const UvFreq F = freqs[e.freq];
  const double stepbw = rsl * F.chanbw;
  const int cr = c % rsl, cs = c / rsl, nsteps = F.nchan / rsl;
  const double f1 = F.lsb ? -(double)(rsl - (cr + 1)) * F.chanbw : cr * F.chanbw;
  const double f2 = F.lsb ? -(double)(nsteps - (cs + 1)) * stepbw : cs * stepbw;
  for (int s = 0; s < npc; s++) {
    const double d = delays[(size_t)e.baseline * maxpc + s];
    float2 out = v;
    if (fabs(d) > 1.0e-20) {
      double edgeturns = d * F.lofreq;
      edgeturns -= floor(edgeturns);
      const double t1 = d * f1 + edgeturns, t2 = d * f2;
      const float a1 = (float)((t1 - floor(t1)) * GX_TWO_PI), a2 = (float)((t2 - floor(t2)) * GX_TWO_PI);
      float s1, c1, s2, c2;
      sincosf(a1, &s1, &c1);
      sincosf(a2, &s2, &c2);
      out = cmul_exact(make_float2(c1, s1), v);      // rotator x data
      out = cmul_exact(out, make_float2(c2, s2));    // times the step rotator
    }
    float2 &r = results[e.ro + (size_t)s * e.stride + c];
    r.x += out.x;
    r.y += out.y;
  }
}

cudaError_t uvshift_launch(const UvEntry *ents, int nents, const float2 *acc, int ks, size_t ks_stride, int N,
                           const double *delays, int npc, int maxpc, const UvFreq *freqs, int rsl, float2 *results,
                           cudaStream_t st)
{
  if (nents <= 0) return cudaSuccess;
  if (nents > 65535) return cudaErrorInvalidConfiguration;
  dim3 grid((N + 127) / 128, nents);
  uvshift_kernel<<<grid, 128, 0, st>>>(ents, acc, ks, ks_stride, N, delays, npc, maxpc, freqs, rsl, results);
  return cudaGetLastError();
}

__global__ void copy_floats_kernel(const float *__restrict__ vals, long long n, float *__restrict__ out)
{
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = vals[i];
}

cudaError_t copy_floats_launch(const float *vals, long long n, float *results_f, long long first, cudaStream_t st)
{
  if (n <= 0) return cudaSuccess;
  copy_floats_kernel<<<(unsigned)std::min<long long>((n + 255) / 256, 1024), 256, 0, st>>>(vals, n, results_f + first);
  return cudaGetLastError();
}

// The pulsar bin of a channel (Polyco::getBins, polyco.cpp:196-222): the
// fractional part of the mean phase plus the channel's dispersion offset,
// bin 0 outside [first end, last end), else the bin whose phase range holds it.
__device__ __forceinline__ int pulsar_bin(double avgphase, double dmoff, const double *__restrict__ bp, int nbins)
{
  const double ap = dmoff + avgphase;
  const double m = ap - floor(ap);
  if (m < bp[0] || m >= bp[nbins - 1]) return 0;
  int bin = 0;
  for (int k = nbins - 1; k > 0; k--)
    if (m < bp[k] && m >= bp[k - 1]) bin = k;
  return bin;
}

__global__ void binned_xmac_kernel(const BinEntry *__restrict__ ents, const float2 *__restrict__ spec, int NI, int N,
                                   int nblk, int b0, const double *__restrict__ avgphase,
                                   const double *__restrict__ dmoff, const double *__restrict__ bp, int nbins,
                                   float2 *__restrict__ acc)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  const BinEntry e = ents[blockIdx.y];
  const size_t bstride = (size_t)NI * N;
  const float2 *xa = spec + ((size_t)e.f * nblk * NI + e.a) * N + c;
  const float2 *xb = spec + ((size_t)e.f * nblk * NI + e.b) * N + c;
  const double dm = dmoff[(size_t)e.f * N + c];
  float2 *row = acc + (size_t)blockIdx.y * nbins * N + c;
  // the current bin's accumulator is carried in registers: the same additions,
  // in block order, as adding into it in memory block by block (core.cpp:943-950)
  int cur = -1;
  float2 sum = make_float2(0.f, 0.f);
  for (int k = 0; k < nblk; k++) {
    const int bin = pulsar_bin(avgphase[b0 + k], dm, bp, nbins);
    if (bin != cur) {
      if (cur >= 0) row[(size_t)cur * N] = sum;
      cur = bin;
      sum = row[(size_t)cur * N];
    }
    const float2 x1 = xa[k * bstride], x2 = xb[k * bstride];
    const float2 p = cmul_exact(x1, make_float2(x2.x, -x2.y));   // vis1 x conj(vis2) (vectorMul_cf32)
    sum.x = __fadd_rn(sum.x, p.x);
    sum.y = __fadd_rn(sum.y, p.y);
  }
  if (cur >= 0) row[(size_t)cur * N] = sum;
}

cudaError_t binned_xmac_launch(const BinEntry *ents, int nents, const float2 *spec, int NI, int N, int nblk, int b0,
                               const double *avgphase, const double *dmoff, const double *binphases, int nbins,
                               float2 *acc, cudaStream_t st)
{
  if (nents <= 0 || nblk <= 0) return cudaSuccess;
  if (nents > 65535) return cudaErrorInvalidConfiguration;
  dim3 grid((N + 127) / 128, nents);
  binned_xmac_kernel<<<grid, 128, 0, st>>>(ents, spec, NI, N, nblk, b0, avgphase, dmoff, binphases, nbins, acc);
  return cudaGetLastError();
}

// One thread per (item, bin); the scrunched sum is bin 0's thread.
__global__ void binned_weights_kernel(const BinWeightItem *__restrict__ items, int nitems, const float *__restrict__ w,
                                      int nblk, int b0, int N, int nbuf, int xstride, const double *__restrict__ avgphase,
                                      const double *__restrict__ dmoff, const double *__restrict__ bp,
                                      const double *__restrict__ bw, int nbins, int scrunch, float *__restrict__ wbins)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int fj = t / nbins, mybin = t % nbins;
  if (fj >= nitems || (scrunch && mybin != 0)) return;
  const BinWeightItem it = items[fj];
  const double *dm = dmoff + (size_t)it.f * N;
  float acc = wbins[t];
  const int nstr = (N + xstride - 1) / xstride;
  // buffered-FFT groups of the subint (core.cpp:784-800), xmac strides, blocks, channels
  for (int g0 = 0; g0 < nblk; g0 += nbuf) {
    const int g1 = min(nblk, g0 + nbuf);
    for (int x = 0; x < nstr; x++) {
      const int c0 = x * xstride, c1 = min(N, c0 + xstride);
      for (int k = g0; k < g1; k++) {
        const float bweight = w[(size_t)it.s1 * nblk + k] * w[(size_t)it.s2 * nblk + k] / N;
        const double ap = avgphase[b0 + k];
        for (int c = c0; c < c1; c++) {
          const int bin = pulsar_bin(ap, dm[c], bp, nbins);
          if (scrunch) {
            if (bw[bin] > 0.0) acc = (float)((double)acc + bweight * bw[bin]);
          } else if (bin == mybin) {
            acc = __fadd_rn(acc, bweight);
          }
        }
      }
    }
  }
  wbins[t] = acc;
}

cudaError_t binned_weights_launch(const BinWeightItem *items, int nitems, const float *w, int nblk, int b0, int N,
                                  int nbuf, int xmacstride, const double *avgphase, const double *dmoff,
                                  const double *binphases, const double *binweights, int nbins, int scrunch,
                                  float *wbins, cudaStream_t st)
{
  if (nitems <= 0 || nblk <= 0) return cudaSuccess;
  const int n = nitems * nbins;
  binned_weights_kernel<<<(n + 63) / 64, 64, 0, st>>>(items, nitems, w, nblk, b0, N, nbuf, xmacstride, avgphase, dmoff,
                                                      binphases, binweights, nbins, scrunch, wbins);
  return cudaGetLastError();
}

__global__ void binned_finalise_kernel(const BinEntry *__restrict__ ents, const float2 *__restrict__ acc, int N,
                                       int nbins, int scrunch, const double *__restrict__ bw,
                                       float2 *__restrict__ results)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  const BinEntry e = ents[blockIdx.y];
  const float2 *row = acc + (size_t)blockIdx.y * nbins * N + c;
  if (!scrunch) {
    for (int b = 0; b < nbins; b++) results[e.ro + (size_t)(b * e.npol + e.p) * N + c] = row[(size_t)b * N];
    return;
  }
  // each bin scaled by its (FP32) weight, then added in bin order (core.cpp:1439-1470, 1808-1823)
  float2 s = make_float2(0.f, 0.f);
  for (int b = 0; b < nbins; b++) {
    const float wf = (float)bw[b];
    const float2 v = row[(size_t)b * N];
    s.x = __fadd_rn(s.x, __fmul_rn(v.x, wf));
    s.y = __fadd_rn(s.y, __fmul_rn(v.y, wf));
  }
  results[e.ro + (size_t)e.p * N + c] = s;
}

__global__ void binned_weights_out_kernel(const BinWeightOut *__restrict__ wo, int n, const float *__restrict__ wbins,
                                          int nbins, float *__restrict__ results_f)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const BinWeightOut x = wo[i];
  results_f[x.float_index] = wbins[(size_t)x.fj * nbins + x.bin];
}

cudaError_t binned_finalise_launch(const BinEntry *ents, int nents, const float2 *acc, int N, int nbins, int scrunch,
                                   const double *binweights, const BinWeightOut *wout, int nwout, const float *wbins,
                                   float2 *results, cudaStream_t st)
{
  if (nents > 65535) return cudaErrorInvalidConfiguration;
  if (nents > 0) {
    dim3 grid((N + 127) / 128, nents);
    binned_finalise_kernel<<<grid, 128, 0, st>>>(ents, acc, N, nbins, scrunch, binweights, results);
  }
  if (nwout > 0)
    binned_weights_out_kernel<<<(nwout + 255) / 256, 256, 0, st>>>(wout, nwout, wbins, nbins,
                                                                   reinterpret_cast<float *>(results));
  return cudaGetLastError();
}

// Channel averaging of the finished result array (Mode::averageFrequency,
// mode.cpp:1376-1401, for autocorrelations; Core's averaged copy,
// core.cpp:1819-1869, for cross products): one CTA per record.
__global__ void average_kernel(const AvgEntry *__restrict__ tab, const float2 *__restrict__ full,
                               float2 *__restrict__ out)
{
  const AvgEntry e = tab[blockIdx.x];
  for (int c = threadIdx.x; c < e.n; c += blockDim.x) {
    const float2 *p = full + e.src + (long long)c * e.L;
    float2 acc = p[0];
    for (int i = 1; i < e.L; i++) {
      acc.x += p[i].x;
      acc.y += p[i].y;
    }
    out[e.dst + c] = e.L == 1 ? acc : make_float2(acc.x / (float)e.L, acc.y / (float)e.L);   // the mean
  }
}

cudaError_t average_launch(const AvgEntry *tab, int nent, const float2 *full, float2 *out, cudaStream_t st)
{
  if (nent <= 0) return cudaSuccess;
  average_kernel<<<nent, 128, 0, st>>>(tab, full, out);
  return cudaGetLastError();
}

}  // namespace gx
