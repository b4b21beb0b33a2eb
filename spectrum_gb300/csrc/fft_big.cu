// fft_big.cu — transforms of 2^19, 2^20 and 2^21 points (the precision
// workload's 2^20-point beams; 2^21 = the reference's nextPow2(2^20) x
// repeat_count 2), beyond what one cluster holds on chip.
//
// nfft = Cb * M, n = M*n1 + n2, k = k1 + Cb*k2:
//   launch 1 (big_cols_kernel): for each n2, the Cb-point DFT over n1 of the
//     windowed, zero-padded samples, times W_N^{n2 k1}, written to scratch[beam][k1][n2] (device memory);
//   2^19 and 2^20 (M = 4096, Cb = 128 or 256): launch 2 (big_rows4_kernel)
//     transforms four rows k1 = 4r .. 4r+3 per CTA and writes bins
//     4r .. 4r+3 + Cb*k2 of the output in the requested mode: runs of four
//     bins, one 32-byte sector, so no separate reordering pass;
//   2^21 (M = 16384, Cb = 128): launch 2 (big_rows_kernel) transforms row k1
//     and writes X[k1 + Cb*k2] back over the row it read; launch 3
//     (rows_transpose_kernel, fft_kernels.cu) writes bin order in the
//     requested mode in contiguous runs (a 16384-point row per CTA leaves no
//     room for four rows, and stride-Cb stores straight from the row kernel
//     kept its SMs waiting on the store queue: 0.63 ms for 64 x 2^20 points).
// Both kernels run in packed arithmetic (fft_pair.cuh).  Measured, complex
// output: 64 x 2^20 0.581 -> 0.467 ms (columns 0.317 -> 0.221, bound by the
// latency of their loads at 15 warps per SM; rows 0.259 -> 0.234, one CTA per
// SM whose phases do not overlap), 64 x 2^19 0.257 -> 0.222, 16 x 2^21 0.393 ->
// 0.342.  Not kept: 32-byte stores per thread in the row kernel (32 x 2^20
// 0.269 -> 0.294), five column CTAs per SM (96 registers, spills: 0.305).
// All twiddles are FP64-generated and stored in FP32, which is what the
// 120 dB dynamic range of the precision workload needs: W_N^{n2 k1}, k1 =
// a + 16 b, as the product of two factor tables [a][n2] = W_N^{n2 a} and
// [b][n2] = W_N^{16 n2 b} (a CTA's slice of the second is read by all its warps from L1,
// where the full [k1][n2] table of nfft entries came from L2); W_M from the local plan.  Replaces hipFFT's internal
// multi-pass plan for large sizes (src/fft_func/src/fft_processor_rocm.cpp:176-193).
#include <algorithm>
#include <cmath>
#include <vector>

#include "fft_core.cuh"
#include "fft_pair.cuh"
#include "spx_internal.h"

namespace spx {

constexpr uint32_t kBigM = 16384;     // row length of the 2^21-point transform
constexpr uint32_t kBigM4 = 4096;     // row length of the 2^19 / 2^20-point transforms
constexpr uint32_t kRows4 = 4;        // rows per CTA of big_rows4_kernel
constexpr int kCols256 = 16;          // columns per CTA of the 256-point column DFTs (32 KB tiles, four per SM)

// Row length M of a big transform of nfft points.
static uint32_t big_rows(uint32_t nfft) { return nfft <= (1u << 20) ? kBigM4 : kBigM; }

// One CTA = W consecutive n2 columns x Cb rows (n1); thread (p, t): column pair
// p < W / 2 (packed arithmetic, fft_pair.cuh), row group t < G; rows of M points.
// Cb = G x J: stage 1 is the J-point DFT over rows t + G j, on samples loaded
// straight into registers (J 16-byte loads in flight per thread); the shared
// tile [Cb][W / 2] of 16-byte slots only carries stage 1's outputs to stage 2,
// the G-point DFT over t.
template <int CB, int G, int W>
__global__ void __launch_bounds__(W / 2 * G, 512 / (W / 2 * G))
big_cols_kernel(const float2* __restrict__ in, uint32_t n_point, const float* __restrict__ win,
                const float2* __restrict__ twN, uint32_t nfft, float2* __restrict__ scratch,
                uint32_t ahead, uint32_t M) {
  extern __shared__ float4 s4[];
  constexpr uint32_t HP = W / 2, T = HP * G;
  const uint32_t tid = threadIdx.x, p = tid % HP, t = tid / HP;
  const uint32_t beam = blockIdx.y, c0 = blockIdx.x * W;
  let_next_launch_begin();
  {  // L2 prefetch of the tile of the CTA `ahead` places later
    const uint64_t f = (uint64_t)blockIdx.y * gridDim.x + blockIdx.x + ahead;
    if (ahead && f < (uint64_t)gridDim.x * gridDim.y) {
      const uint32_t fb = (uint32_t)(f / gridDim.x), fc = (uint32_t)(f % gridDim.x) * W;
      for (uint32_t r = tid; r < CB; r += T) {
        const uint32_t lo = r * M + fc, hi = min(lo + W, n_point);
        if (lo < hi) prefetch_l2(in + (size_t)fb * n_point + lo, (size_t)(hi - lo) * sizeof(float2), 0, 1);
      }
    }
  }
  constexpr int J = CB / G;  // stage-1 radix
  static_assert(J == 16, "the W_N factor tables are built for k1 = a + 16 b");
  const uint32_t n2 = c0 + 2 * p;
  // stage 1: thread t transforms rows t + G j (j < J), twiddles W_CB^{t a}
  C2 v[J];
  SamplePairs(in + (size_t)beam * n_point, n_point, win).load(v, t * M + n2, G * M);
  PDft<J>::run(v);
#pragma unroll
  for (int a = 0; a < J; ++a) {
    if (a > 0) {
      const float2 w = __ldg(twN + (size_t)(J + G) * M + (t * a) % CB);  // W_CB^e, after the two factor tables
      v[a] = c2mul(v[a], C2{pk(w.x), pk(w.y)});
    }
    s4[(t + G * a) * HP + p] = make_float4(v[a].x.x, v[a].x.y, v[a].y.x, v[a].y.y);
  }
  __syncthreads();
  // stage 2: for a = t, t + G, ... (< J), the G-point DFT over t' of rows t' + G a -> k1 = a + J b
  auto pair_tw = [&](uint32_t row) {  // W_N factor of columns n2, n2 + 1
    const float4 w = __ldg(reinterpret_cast<const float4*>(twN + (size_t)row * M + n2));
    return C2{make_float2(w.x, w.z), make_float2(w.y, w.w)};
  };
  float2* o = scratch + (size_t)beam * nfft + n2;
#pragma unroll 1
  for (uint32_t a = t; a < (uint32_t)J; a += G) {
    C2 w[G];
#pragma unroll
    for (int tp = 0; tp < G; ++tp) {
      const float4 z = s4[(tp + G * a) * HP + p];
      w[tp] = C2{make_float2(z.x, z.y), make_float2(z.z, z.w)};
    }
    PDft<G>::run(w);
    const C2 ta = pair_tw(a);  // W_N^{n2 a}
#pragma unroll
    for (int b = 0; b < G; ++b) {  // k1 = a + J b: W_N^{n2 k1} = W_N^{n2 a} W_N^{n2 J b}
      const C2 z = c2mul(w[b], c2mul(ta, pair_tw(J + b)));
      __stcg(reinterpret_cast<float4*>(o + (size_t)(a + J * b) * M), make_float4(z.x.x, z.y.x, z.x.y, z.y.y));
    }
  }
}

// Rows of 16384 points (2^21), each written back over itself.
__global__ void __launch_bounds__(512, 1)
big_rows_kernel(FftGeom g, const float4* __restrict__ tw_pair, float2* __restrict__ scratch) {
  extern __shared__ float4 s4[];
  const uint32_t tid = threadIdx.x;
  float2* row = scratch + (size_t)blockIdx.x * g.M;
  if (g.ahead && blockIdx.x + g.ahead < gridDim.x)  // the row the CTA one wave later reads
    prefetch_l2(row + (size_t)g.ahead * g.M, (size_t)g.M * sizeof(float2), tid, 512);
  // the row is read by this CTA alone (first pass, before its barrier)
  pair_local_fft_out<(int)kBigM>(s4, ExchangePairs<>{row}, tw_pair, tid, RowOutPairs{row});
}

// Four rows k1 = r0 .. r0+3 of 4096 points per CTA in packed arithmetic
// (fft_pair.cuh).  The first two passes run one row per group of 128 threads
// behind the group's own barriers; in the last one the rows are interleaved
// over the lanes (thread (q, t): row r0 + q, butterflies 2t, 2t + 1), so its
// registers hold one element of neighbouring rows in neighbouring lanes and go
// out in the requested mode as runs of four bins, 32-byte sectors.  Row pitch
// in slots: the four lanes of one element and two neighbouring slots of each
// hit eight different 16-byte banks.
constexpr uint32_t kRowPitch4 = ps_len(kBigM4) + 2;
constexpr int kBigComplex = 0, kBigMag = 1, kBigMagPhase = 2, kBigOther = 3, kBigReversed = 4, kBigHalf = 5;

template <int MODE, bool LAST = false>
__global__ void __launch_bounds__(kRows4 * 128, 1)
big_rows4_kernel(FftGeom g, const float4* __restrict__ tw_pair, const float2* cols,
                 void* __restrict__ out, uint32_t out_mode, float scale) {
  extern __shared__ float4 s4[];
  constexpr int TG = 128, M = (int)kBigM4;
  const uint32_t tid = threadIdx.x, grp = tid / TG;
  const uint32_t per_beam = g.C / kRows4;
  const uint32_t beam = blockIdx.x / per_beam, r0 = (blockIdx.x - beam * per_beam) * kRows4;
  const float2* scratch = wait_for_launch_before(cols);
  const float2* row = scratch + (size_t)beam * g.nfft + (size_t)(r0 + grp) * kBigM4;
  // the four rows of the CTA one residency wave later follow this CTA's
  // (CTA b holds elements [b, b + 1) x kRows4 x kBigM4 of the scratch)
  if (g.ahead && blockIdx.x + g.ahead < gridDim.x)
    prefetch_l2(scratch + (size_t)(blockIdx.x + g.ahead) * (kRows4 * kBigM4), kRows4 * kBigM4 * sizeof(float2), tid,
                kRows4 * TG);
  float4* s = s4 + grp * kRowPitch4;
  pair_first<M, TG, GroupSync<TG>>(s, ExchangePairs<LAST>{row}, tid - grp * TG);
  pair_passes_until_last<M, 1, TG, GroupSync<TG>>(s, tw_pair, tid - grp * TG);
  __syncthreads();
  const uint32_t q = tid % kRows4, k1 = r0 + q;
  float4* sq = s4 + q * kRowPitch4;
  if constexpr (MODE == kBigOther) {
    // mirrored real-input spectra: through shared memory, the general output
    // function having no room beside the last pass's registers
    pair_last<M, TG>(sq, tw_pair, tid / kRows4, SlotOut{sq});
    __syncthreads();
#pragma unroll 4
    for (uint32_t p = tid / kRows4; p < kBigM4 / 2; p += TG) {
      const float4 z = sq[ps(p)];
      store_bin(out, out_mode, scale, g, beam, k1 + g.C * (2 * p), make_float2(z.x, z.z));
      store_bin(out, out_mode, scale, g, beam, k1 + g.C * (2 * p + 1), make_float2(z.y, z.w));
    }
  } else {
    pair_last<M, TG>(sq, tw_pair, tid / kRows4, [&](uint32_t e, C2 z) {
      const size_t at = (size_t)beam * g.nfft + k1 + (size_t)g.C * e;
      const float2 a = first_of(z), b = second_of(z);
      if constexpr (MODE == kBigComplex) {
        reinterpret_cast<float2*>(out)[at] = a;
        reinterpret_cast<float2*>(out)[at + g.C] = b;
      } else if constexpr (MODE == kBigMagPhase) {
        // one phase after another: their registers would not fit side by side (through
        // shared memory instead, 64 x 2^19 points 270 us for 263)
        float2* o = reinterpret_cast<float2*>(out) + at;
        o[0] = make_float2(mag_rn(a), atan2f(a.y, a.x));
        asm volatile("" ::: "memory");
        o[g.C] = make_float2(mag_rn(b), atan2f(b.y, b.x));
        asm volatile("" ::: "memory");
      } else if constexpr (MODE == kBigHalf) {
        const uint32_t k = k1 + g.C * e, half = g.nfft / 2;
        float2* o = reinterpret_cast<float2*>(out) + (size_t)beam * (half + 1) + k;
        if (k <= half) o[0] = a;
        if (k + g.C <= half) o[g.C] = b;
      } else if constexpr (MODE == kBigReversed) {
        const uint32_t k = k1 + g.C * e;
        float2* o = reinterpret_cast<float2*>(out) + (size_t)beam * g.nfft;
        o[(g.nfft - k) & (g.nfft - 1)] = make_float2(__fmul_rn(a.x, scale), __fmul_rn(a.y, scale));
        o[g.nfft - k - g.C] = make_float2(__fmul_rn(b.x, scale), __fmul_rn(b.y, scale));
      } else {
        float* o = reinterpret_cast<float*>(out);
        const float a2 = mag2_rn(a), b2 = mag2_rn(b);
        o[at] = __fmul_rn(out_mode == SPX_OUT_MAG2 ? a2 : __fsqrt_rn(a2), scale);
        o[at + g.C] = __fmul_rn(out_mode == SPX_OUT_MAG2 ? b2 : __fsqrt_rn(b2), scale);
      }
    });
  }
}

bool big_size(uint32_t nfft) { return nfft == (1u << 19) || nfft == (1u << 20) || nfft == (1u << 21); }

// Geometry of the row FFTs (M points, C = Cb as the output stride) and the
// W_N table; called by get_plan for big sizes.
spx_status build_big_plan(spx_ctx* ctx, uint32_t nfft, FftPlan* plan) {
  const uint32_t M = big_rows(nfft);
  FftGeom gl{};
  if (!build_geom(M, &gl, kEPTDefault)) return fail(ctx, SPX_ERR_INVALID_ARG, "big plan");
  gl.nfft = nfft;
  gl.C = nfft / M;
  plan->g = gl;
  plan->big = true;
  std::vector<float2> twl(M);
  fill_local_twiddles(gl, twl.data());
  // W_N^{n2 k1} for k1 = a + 16 b as two factor tables, [a][n2] = W_N^{n2 a}
  // (a < 16) and [16 + b][n2] = W_N^{16 n2 b} (b < Cb / 16), then the Cb
  // entries W_Cb^e = W_N^{e M}
  const uint32_t cb = gl.C, J = 16, G = cb / J;
  std::vector<float2> twn((size_t)(J + G) * M + cb);
  auto w_n = [nfft](uint64_t m) {
    m %= nfft;
    const double a = -2.0 * M_PI * (double)m / (double)nfft;
    return make_float2((float)std::cos(a), (float)std::sin(a));
  };
  for (uint32_t a = 0; a < J; ++a)
    for (uint32_t n2 = 0; n2 < M; ++n2) twn[(size_t)a * M + n2] = w_n((uint64_t)n2 * a);
  for (uint32_t b = 0; b < G; ++b)
    for (uint32_t n2 = 0; n2 < M; ++n2) twn[(size_t)(J + b) * M + n2] = w_n((uint64_t)n2 * J * b);
  for (uint32_t e = 0; e < cb; ++e) twn[(size_t)(J + G) * M + e] = w_n((uint64_t)e * M);
  cudaError_t e = cudaMalloc(&plan->d_tw_local, twl.size() * sizeof(float2));
  if (e == cudaSuccess) e = cudaMemcpy(plan->d_tw_local, twl.data(), twl.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = upload_pair_twiddles(plan, twl.data());
  if (e == cudaSuccess) e = cudaMalloc(&plan->d_tw_cross, twn.size() * sizeof(float2));
  if (e == cudaSuccess) e = cudaMemcpy(plan->d_tw_cross, twn.data(), twn.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "big plan tables");
  return SPX_OK;
}

spx_status launch_fft_big(spx_ctx* ctx, const FftPlan& plan, const float2* d_in, uint32_t beams,
                          uint32_t n_point, const float* d_win, uint32_t out_mode, float scale,
                          void* d_out) {
  if (beams == 0) return SPX_OK;
  const FftGeom& g = plan.g;
  void* scr = nullptr;
  spx_status st = get_scratch(ctx, kSlotExchange, (size_t)beams * g.nfft * sizeof(float2), &scr);
  if (st != SPX_OK) return st;
  float2* scratch = static_cast<float2*>(scr);
  const uint32_t M = g.M;
  // Cb = 128 (2^19 as 128 x 4096, 2^21 as 128 x 16384: 8 x 16) or 256 (2^20
  // as 256 x 4096: 16 x 16)
  const uint32_t W = g.C == 256 ? kCols256 : 32u, cthreads = W / 2 * (g.C / 16);
  const void* kcols = g.C == 256 ? (const void*)big_cols_kernel<256, 16, kCols256>
                                 : (const void*)big_cols_kernel<128, 8, 32>;
  const size_t csmem = (size_t)g.C * W * sizeof(float2);
  cudaError_t e = configure_kernel(kcols, csmem);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "configure big_cols_kernel");
  const uint32_t ahead_cols = ctx->input_on_host ? 0u : resident_ctas(kcols, cthreads, csmem, 1);
  void* cargs[] = {(void*)&d_in, (void*)&n_point, (void*)&d_win, (void*)&plan.d_tw_cross, (void*)&g.nfft,
                   (void*)&scratch, (void*)&ahead_cols, (void*)&M};
  e = cudaLaunchKernel(kcols, dim3(M / W, beams), dim3(cthreads), cargs, csmem, ctx->stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "launch big_cols_kernel");
  const float4* twp = plan.d_tw_pair;
  FftGeom gg = g;
  gg.beams = beams;
  if (M == kBigM4) {  // four rows per CTA, bin order written directly
    // While the scratch and a complex spectrum fit L2 together (129 MB), the scratch
    // leaves it as it is read: else the spectrum is driven out, and a search behind
    // the transform is slower (top-5 of 8 x 2^20 points 565 -> 478 us, of 16 x 2^19
    // 320 -> 274; the spectra alone 74.5 -> 73.5).  From 96 MB of scratch on, 1 .. 5 %
    // slower that way.
    const bool last = (size_t)beams * g.nfft * sizeof(float2) <= (64u << 20);
    const void* kfn = out_mode == SPX_OUT_COMPLEX ? (last ? (const void*)big_rows4_kernel<kBigComplex, true>
                                                          : (const void*)big_rows4_kernel<kBigComplex>)
                      : out_mode == SPX_OUT_MAG || out_mode == SPX_OUT_MAG2
                          ? (const void*)big_rows4_kernel<kBigMag>
                      : out_mode == SPX_OUT_MAGPHASE    ? (const void*)big_rows4_kernel<kBigMagPhase>
                      : out_mode == kOutComplexReversed ? (const void*)big_rows4_kernel<kBigReversed>
                      : out_mode == kOutR2CHalf         ? (const void*)big_rows4_kernel<kBigHalf>
                                                        : (const void*)big_rows4_kernel<kBigOther>;
    const size_t smem = (size_t)kRows4 * kRowPitch4 * sizeof(float4);
    e = configure_kernel(kfn, smem);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "configure big_rows4_kernel");
    gg.ahead = ctx->input_on_host ? 0u : resident_ctas(kfn, kRows4 * 128, smem, 1);
    const float2* scr_c = scratch;
    void* args[] = {(void*)&gg, (void*)&twp, (void*)&scr_c, (void*)&d_out, (void*)&out_mode, (void*)&scale};
    e = launch_dependent(kfn, dim3(beams * (g.C / kRows4)), dim3(kRows4 * 128), args, smem, ctx->stream);
    return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, "launch big_rows4_kernel");
  }
  const void* kfn = (const void*)big_rows_kernel;
  const size_t smem = ps_len(kBigM) * sizeof(float4);
  e = configure_kernel(kfn, smem);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "configure big_rows_kernel");
  gg.ahead = resident_ctas(kfn, 512, smem, 1);
  void* args[] = {(void*)&gg, (void*)&twp, (void*)&scratch};
  e = cudaLaunchKernel(kfn, dim3(beams * g.C), dim3(512), args, smem, ctx->stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "launch big_rows_kernel");
  return launch_rows_transpose(ctx, g, scratch, beams, d_out, out_mode, scale);
}

}  // namespace spx
