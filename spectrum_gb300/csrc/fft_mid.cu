// fft_mid.cu — transforms of C x 16384 points (32768, 49152, 65536 .. 262144)
// in two launches of small CTAs.
//
// The plan is that of the beam groups (fft_core.cuh): nfft = C x 16384 with a
// C-point cross stage, then a 16384-point local FFT of radices 16, 16, 16, 4;
// the operations and twiddles of every element are the same, so the spectra
// are the same bits.  What changes is where the data crosses device memory:
// after the local FFT's FIRST radix-16 pass instead of before it.
//   n = 16384 n1 + 1024 r + j,  k = k1 + C (r0 + 16 kr)
//   launch 1 (mid_cols_kernel): for each column j, the C-point DFTs over n1 of
//     the windowed, zero-padded samples, times W_N^{(1024 r + j) k1}, then the
//     16-point DFTs over r: row rho = k1 + C r0 of the scratch, element j;
//   launch 2 (mid_rows_kernel): the remaining passes (16, 16, 4 with strides
//     16, 256, 4096) act on each row alone: a 1024-point FFT over j whose
//     twiddles depend on r0, one warp per row and four rows per CTA; bin
//     rho + 16 C kr of the spectrum is element kr of row rho, so four rows
//     give runs of four bins (one 32-byte sector) in bin order.
//
// Why: the 16384-point local FFT takes the whole register file and 136 KB of
// shared memory of an SM, so its load, exchange and store phases never overlap
// (ncu: 22 400 cycles per row against ~7 000 of issue and ~7 000 of
// shared-memory traffic).  Tiles of 4096 points leave five CTAs per SM in
// different phases, the rows need only warp barriers, the twiddles of a row fit
// L1, and the spectrum comes out in bin order without a transpose.
// 256 beams of 65536 samples in 131072 bins: launch 1 0.065 ms (6.2 TB/s of
// samples and scratch), bound by device memory and load latency; launch 2 0.066 ms
// (6.0 TB/s), bound by the L1's data path (77 % of its wavefronts: two exchanges,
// twiddles, loads).  In bin order launch 2 takes 0.12 ms: runs of four bins cost the
// L1 as much as the rest.
//
// Replaces hipfftExecC2C's multi-pass plans
// (src/fft_func/src/fft_processor_rocm.cpp:176-193).
#include <algorithm>
#include <cmath>
#include <vector>

#include "fft_core.cuh"
#include "fft_pair.cuh"
#include "spx_internal.h"

namespace spx {

constexpr uint32_t kMidLocal = 16384;  // local size of the plan
constexpr uint32_t kMidRow = 1024;     // row length of launch 2

// Twiddles of a row with index r0, in float4 entries:
//   [0, 8)     W_256^{r r0}, r < 16, two complex values to an entry (stride 16)
//   [16, 136)  W_4096^{r k}, k = 16 q + r0, pairs q, q + 1 at [(r - 1) 8 + q/2] (stride 256)
//   [136, 138) W_16384^{16 (q mod 4) + r0}, pairs; [138, 202) W_16384^{64 j} twice over (stride 4096)
constexpr uint32_t kMidTw = 208;

// ---- launch 1 ----------------------------------------------------------------------
// Thread groups per column pair: C, rounded up to a power of two.
template <int C>
constexpr int kMidGroups = C <= 2 ? 2 : C <= 4 ? 4 : C <= 8 ? 8 : 16;
// Columns per CTA: 128 threads (256 for 16 groups, whose rows of 32 columns
// keep 256-byte runs).
template <int C>
constexpr int kMidCols = kMidGroups<C> == 16 ? 32 : 256 / kMidGroups<C>;

// Thread (p, g): column pair p, group g < G.  Stage 1: rows r = g + G u
// (u < 16 / G), the C-point DFT over n1 and its twiddles; stage 2: k1 = g < C,
// the 16-point DFT over r.  All loads of a thread (16 bytes each) are issued
// before its first DFT.  Slots of the tile are [k1][r][p]: every access of a
// warp is contiguous.
// CHIRP: the samples of a chirp-z transform, times its chirp.
template <int C, bool CHIRP>
__global__ void __launch_bounds__(kMidCols<C> / 2 * kMidGroups<C>, kMidGroups<C> == 16 ? 2 : C == 2 || CHIRP ? 4 : 5)
mid_cols_kernel(const float2* __restrict__ in, uint32_t n_point, const float* __restrict__ win,
                const float2* __restrict__ twc, float2* __restrict__ scratch, uint32_t ahead,
                const float2* __restrict__ chirp) {
  extern __shared__ float4 s4[];
  constexpr uint32_t W = kMidCols<C>, HP = W / 2, G = kMidGroups<C>, U = 16 / G, nfft = C * kMidLocal;
  const uint32_t tid = threadIdx.x, p = tid % HP, g = tid / HP;
  const uint32_t beam = blockIdx.x / (kMidRow / W), c0 = (blockIdx.x - beam * (kMidRow / W)) * W;
  let_next_launch_begin();
  if (ahead && blockIdx.x + ahead < gridDim.x) {  // L2 prefetch of the tile one residency wave later
    const uint32_t f = blockIdx.x + ahead, fb = f / (kMidRow / W), fc = (f - fb * (kMidRow / W)) * W;
    for (uint32_t r = tid; r < 16 * C; r += HP * G) {
      const uint32_t lo = r * kMidRow + fc, hi = min(lo + W, n_point);
      if (lo < hi) prefetch_l2(in + (size_t)fb * n_point + lo, (size_t)(hi - lo) * sizeof(float2), 0, 1);
    }
  }
  const SamplePairs ld(in + (size_t)beam * n_point, n_point, win);
  const uint32_t j = c0 + 2 * p;
  C2 v[U][C];
#pragma unroll
  for (uint32_t u = 0; u < U; ++u) {
    if constexpr (CHIRP)
      ChirpPairs{ld, chirp}.load(v[u], kMidRow * (g + G * u) + j, kMidLocal);
    else
      ld.load(v[u], kMidRow * (g + G * u) + j, kMidLocal);
  }
#pragma unroll
  for (uint32_t u = 0; u < U; ++u) {
    const uint32_t r = g + G * u;
    const float4 t = __ldg(reinterpret_cast<const float4*>(twc + kMidRow * r + j));
    PDft<C>::run(v[u]);
    C2 w[C];
    w[1] = C2{make_float2(t.x, t.z), make_float2(t.y, t.w)};
#pragma unroll
    for (int k1 = 2; k1 < C; ++k1) w[k1] = (k1 % 2 == 0) ? c2mul(w[k1 / 2], w[k1 / 2]) : c2mul(w[k1 - 1], w[1]);
#pragma unroll
    for (int k1 = 0; k1 < C; ++k1) {
      const C2 z = k1 == 0 ? v[u][0] : c2mul(v[u][k1], w[k1]);
      s4[(k1 * 16 + r) * HP + p] = make_float4(z.x.x, z.x.y, z.y.x, z.y.y);
    }
  }
  __syncthreads();
  if (C < (int)G && g >= (uint32_t)C) return;
  C2 b[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    const float4 a = s4[(g * 16 + r) * HP + p];
    b[r] = C2{make_float2(a.x, a.y), make_float2(a.z, a.w)};
  }
  PDft<16>::run(b);
  float2* o = scratch + (size_t)beam * nfft + g * kMidRow + j;
#pragma unroll
  for (int r0 = 0; r0 < 16; ++r0)
    __stcg(reinterpret_cast<float4*>(o + r0 * (C * kMidRow)),
           make_float4(b[r0].x.x, b[r0].y.x, b[r0].x.y, b[r0].y.y));
}

// ---- launch 2 ----------------------------------------------------------------------
struct MidRowsArgs {
  FftGeom g;
  const float4* tw;       // [16][kMidTw]
  float2* scratch;
  void* out;
  uint32_t out_mode;
  float scale;
  uint32_t qlo, qhi;      // window form: elements [qlo, qhi) of each row are written
  const float2* chirp;    // chirp-z forms: FFT_m(b), or the chirp
  FftGeom og;             // kMidChirpPost: geometry of the output (its nfft bins)
};
constexpr int kMidComplex = 0, kMidMag = 1, kMidOther = 2;
// Chirp-z forms: times FFT_m(b); bin k is element (m - k) mod m of the
// convolution, scaled by 1/m, times the chirp into the output
constexpr int kMidChirpMul = 3, kMidChirpPost = 4, kMidMagPhase = 5;
constexpr uint32_t kMidRows = 4;  // rows per CTA

struct WarpSync {
  static SPX_DEV void wait() { __syncwarp(); }
};

// The passes of CtPlan<1024> (16, 16, 4) in row coordinates with the row's
// twiddles tw, by 32 threads t = 0 .. 31 that share the slots s;
// out(q, z) takes elements q, q + 1 (q even) of the result.
template <typename Sync, typename Out>
SPX_DEV void mid_row_fft(float4* s, const float2* row, const float4* __restrict__ tw, uint32_t t, const Out& out) {
  {
    C2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const float4 x = __ldcs(reinterpret_cast<const float4*>(row + 2 * t + 64 * r));
      v[r] = C2{make_float2(x.x, x.z), make_float2(x.y, x.w)};
    }
    // one twiddle for the whole row: 8-byte loads (a 16-byte load costs the L1
    // four write-back cycles, an 8-byte one two)
    const float2* w1 = reinterpret_cast<const float2*>(tw);
#pragma unroll
    for (int r = 1; r < 16; ++r) {
      const float2 w = __ldg(w1 + r);
      v[r] = c2mul(v[r], C2{pk(w.x), pk(w.y)});
    }
    PDft<16>::run(v);
    float4* d = s + 17 * t;
#pragma unroll
    for (int r = 0; r < 16; r += 2) {
      d[r / 2] = make_float4(v[r].x.x, v[r + 1].x.x, v[r].y.x, v[r + 1].y.x);
      d[8 + r / 2] = make_float4(v[r].x.y, v[r + 1].x.y, v[r].y.y, v[r + 1].y.y);
    }
  }
  Sync::wait();
  {
    C2 v[16];
    pair_load<(int)kMidRow, 1>(s, v, t);
    Sync::wait();
    const uint32_t kk = t & 7;
#pragma unroll
    for (int r = 1; r < 16; ++r) v[r] = c2mul(v[r], ld_tw(tw + 16 + (r - 1) * 8 + kk));
    PDft<16>::run(v);
    float4* d = s + ps((t - kk) * 16 + kk);
#pragma unroll
    for (int r = 0; r < 16; ++r) d[r * 8 + (r >> 1)] = make_float4(v[r].x.x, v[r].x.y, v[r].y.x, v[r].y.y);
  }
  Sync::wait();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t m = t + 32 * u;
    C2 v[4];
    pair_load<(int)kMidRow, 2>(s, v, m);
    const C2 w1 = c2mul(ld_tw(tw + 138 + (m >> 1)), ld_tw(tw + 136 + (m & 1)));
    const C2 w2 = c2mul(w1, w1);
    v[1] = c2mul(v[1], w1);
    v[2] = c2mul(v[2], w2);
    v[3] = c2mul(v[3], c2mul(w2, w1));
    PDft<4>::run(v);
#pragma unroll
    for (int r = 0; r < 4; ++r) out(2 * m + 256 * r, v[r]);
  }
}

// Beams in descending order (the rows written last by launch 1 may still be
// in L2), and the L2 prefetch of the rows (contiguous) of the CTA one
// residency wave later.
SPX_DEV uint32_t mid_rows_block(MidRowsArgs& a) {
  let_next_launch_begin();
  a.scratch = wait_for_launch_before(a.scratch);
  const uint32_t bx = gridDim.x - 1 - blockIdx.x;
  if (a.g.ahead && bx >= a.g.ahead && threadIdx.x < kMidRows / 2)
    prefetch_l2(a.scratch + ((size_t)(bx - a.g.ahead) * kMidRows + threadIdx.x * 2) * kMidRow,
                2 * kMidRow * sizeof(float2), 0, 1);
  return bx;
}

// Window form: one warp per row, elements [qlo, qhi) (whole pairs) written
// back over the row it read: coalesced, and no barrier wider than a warp.
__global__ void __launch_bounds__(32 * kMidRows, 4)
mid_rows_window_kernel(MidRowsArgs a) {
  extern __shared__ float4 s4[];
  const uint32_t t = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t CB = 16 * a.g.C;
  const uint32_t rr = mid_rows_block(a) * kMidRows + warp;  // row of the scratch
  float2* row = a.scratch + (size_t)rr * kMidRow;
  const uint32_t r0 = (rr % CB) / a.g.C, qlo = a.qlo, qhi = a.qhi;
  mid_row_fft<WarpSync>(s4 + warp * ps_len(kMidRow), row, a.tw + r0 * kMidTw, t, [=](uint32_t q, C2 z) {
    if (q >= qlo && q < qhi)
      __stcg(reinterpret_cast<float4*>(row + q), make_float4(z.x.x, z.y.x, z.x.y, z.y.y));
  });
}

// Bin-order form.  Thread (q, t): row rho0 + q, pairs of butterflies t.  The
// rows of a CTA are interleaved over the lanes, so the last pass's registers
// hold the same element of neighbouring rows in neighbouring lanes and go out
// as runs of four bins without another trip through shared memory.  Row pitch
// in slots: the four lanes of one element and two neighbouring slots of each
// hit eight different 16-byte banks.  (Eight rows per CTA, runs of 64 bytes but
// loads of half lines: 131072 points 0.233 -> 0.255 ms per 2^25 points.)
constexpr uint32_t kMidPitch = ps_len(kMidRow) + 2;

template <int MODE>
__global__ void __launch_bounds__(32 * kMidRows, 4)
mid_rows_kernel(MidRowsArgs a) {
  extern __shared__ float4 s4[];
  const uint32_t tid = threadIdx.x, q = tid % kMidRows, t = tid / kMidRows;
  const uint32_t C = a.g.C, CB = 16 * C, per_beam = CB / kMidRows;
  const uint32_t bx = mid_rows_block(a);
  const uint32_t beam = bx / per_beam, rho = (bx - beam * per_beam) * kMidRows + q;
  const float2* row = a.scratch + ((size_t)bx * kMidRows + q) * kMidRow;
  mid_row_fft<CtaSync>(s4 + q * kMidPitch, row, a.tw + (rho / C) * kMidTw, t, [=](uint32_t e, C2 zz) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t k = rho + CB * (e + h);
      const float2 z = h ? second_of(zz) : first_of(zz);
      const size_t at = (size_t)beam * a.g.nfft + k;
      if constexpr (MODE == kMidComplex) {
        reinterpret_cast<float2*>(a.out)[at] = z;
      } else if constexpr (MODE == kMidMagPhase) {
        reinterpret_cast<float2*>(a.out)[at] = make_float2(mag_rn(z), atan2f(z.y, z.x));
      } else if constexpr (MODE == kMidChirpMul) {
        reinterpret_cast<float2*>(a.out)[at] = cmul(z, __ldg(a.chirp + k));
      } else if constexpr (MODE == kMidChirpPost) {
        const float inv = 1.0f / (float)a.g.nfft;
        const uint32_t b = (a.g.nfft - k) & (a.g.nfft - 1);
        if (b < a.og.nfft)
          store_bin(a.out, a.out_mode, a.scale, a.og, beam, b,
                    cmul(make_float2(__fmul_rn(z.x, inv), __fmul_rn(z.y, inv)), __ldg(a.chirp + b)));
      } else if constexpr (MODE == kMidMag) {
        const float m2 = mag2_rn(z);
        reinterpret_cast<float*>(a.out)[at] = __fmul_rn(a.out_mode == SPX_OUT_MAG2 ? m2 : __fsqrt_rn(m2), a.scale);
      } else {
        store_bin(a.out, a.out_mode, a.scale, a.g, beam, k, z);
      }
    }
  });
}

// ---- host --------------------------------------------------------------------------
bool mid_geometry(const FftGeom& g) {
  return g.M == kMidLocal && g.ept == 16 && g.C > 1;
}

cudaError_t upload_mid_twiddles(FftPlan* plan, const float2* twl) {
  const FftGeom& g = plan->g;
  if (!mid_geometry(g)) return cudaSuccess;
  // the scalar tables of passes 1 .. 3 (strides 16, 256, 4096)
  const float2 *t1 = twl + g.twoff[1], *t2 = twl + g.twoff[2], *t3 = twl + g.twoff[3];
  std::vector<float4> t(16 * kMidTw, make_float4(0.f, 0.f, 0.f, 0.f));
  auto two = [](float2 a, float2 b) { return make_float4(a.x, b.x, a.y, b.y); };
  for (uint32_t r0 = 0; r0 < 16; ++r0) {
    float4* o = t.data() + r0 * kMidTw;
    float2* o1 = reinterpret_cast<float2*>(o);
    for (uint32_t r = 1; r < 16; ++r) {
      o1[r] = t1[(r - 1) * 16 + r0];
      for (uint32_t q = 0; q < 16; q += 2)
        o[16 + (r - 1) * 8 + q / 2] = two(t2[(r - 1) * 256 + 16 * q + r0], t2[(r - 1) * 256 + 16 * (q + 1) + r0]);
    }
    for (uint32_t h = 0; h < 2; ++h) o[136 + h] = two(t3[32 * h + r0], t3[32 * h + 16 + r0]);
    for (uint32_t j = 0; j < 64; ++j) o[138 + j] = two(t3[64 + j], t3[64 + j]);
  }
  cudaError_t e = cudaMalloc(&plan->d_tw_rows, t.size() * sizeof(float4));
  if (e == cudaSuccess) e = cudaMemcpy(plan->d_tw_rows, t.data(), t.size() * sizeof(float4), cudaMemcpyHostToDevice);
  return e;
}

template <int C>
static cudaError_t launch_cols(spx_ctx* ctx, const FftPlan& plan, const float2* d_in, uint32_t beams,
                               uint32_t n_point, const float* d_win, float2* scratch, const float2* chirp) {
  const void* kfn = (const void*)mid_cols_kernel<C, false>;
  if constexpr ((C & (C - 1)) == 0)  // chirp-z transforms take powers of two
    if (chirp) kfn = (const void*)mid_cols_kernel<C, true>;
  constexpr uint32_t threads = kMidCols<C> / 2 * kMidGroups<C>;
  const size_t smem = (size_t)16 * C * kMidCols<C> * sizeof(float2);
  cudaError_t e = configure_kernel(kfn, smem);
  if (e != cudaSuccess) return e;
  uint32_t ahead = ctx->input_on_host ? 0u : resident_ctas(kfn, threads, smem, 1);
  void* args[] = {(void*)&d_in, (void*)&n_point, (void*)&d_win, (void*)&plan.d_tw_cross, (void*)&scratch, (void*)&ahead,
                  (void*)&chirp};
  return cudaLaunchKernel(kfn, dim3(beams * (kMidRow / kMidCols<C>)), dim3(threads), args, smem, ctx->stream);
}

// Launch 1 into the exchange scratch (with the samples times `chirp` when not
// null), then launch 2 (kernel kfn).
static spx_status launch_mid(spx_ctx* ctx, const FftPlan& plan, const float2* d_in, uint32_t beams, uint32_t n_point,
                             const float* d_win, float2* scratch, const void* kfn, size_t smem, MidRowsArgs a,
                             const float2* chirp = nullptr) {
  cudaError_t e;
  switch (plan.g.C) {
    case 2: e = launch_cols<2>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
    case 3: e = launch_cols<3>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
    case 6: e = launch_cols<6>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
    case 9: e = launch_cols<9>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
    case 12: e = launch_cols<12>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
    case 4: e = launch_cols<4>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
    case 8: e = launch_cols<8>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
    default: e = launch_cols<16>(ctx, plan, d_in, beams, n_point, d_win, scratch, chirp); break;
  }
  if (e != cudaSuccess) return cuda_fail(ctx, e, "launch mid_cols_kernel");
  e = configure_kernel(kfn, smem);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "configure mid_rows_kernel");
  a.g = plan.g;
  a.g.beams = beams;
  a.g.ahead = resident_ctas(kfn, 32 * kMidRows, smem, 1);
  a.tw = plan.d_tw_rows;
  a.scratch = scratch;
  void* args[] = {(void*)&a};
  e = launch_dependent(kfn, dim3(beams * (16 * plan.g.C / kMidRows)), dim3(32 * kMidRows), args, smem, ctx->stream);
  return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, "launch mid_rows_kernel");
}

spx_status launch_fft_mid(spx_ctx* ctx, const FftPlan& plan, const float2* d_in, uint32_t beams, uint32_t n_point,
                          const float* d_win, uint32_t out_mode, float scale, void* d_out) {
  void* scr = nullptr;
  spx_status st = get_scratch(ctx, kSlotExchange, (size_t)beams * plan.g.nfft * sizeof(float2), &scr);
  if (st != SPX_OK) return st;
  MidRowsArgs a{};
  a.out = d_out;
  a.out_mode = out_mode;
  a.scale = scale;
  const void* kfn = out_mode == SPX_OUT_COMPLEX ? (const void*)mid_rows_kernel<kMidComplex>
                    : out_mode == SPX_OUT_MAG || out_mode == SPX_OUT_MAG2
                        ? (const void*)mid_rows_kernel<kMidMag>
                    : out_mode == SPX_OUT_MAGPHASE ? (const void*)mid_rows_kernel<kMidMagPhase>
                                                   : (const void*)mid_rows_kernel<kMidOther>;
  return launch_mid(ctx, plan, d_in, beams, n_point, d_win, static_cast<float2*>(scr), kfn,
                    kMidRows * kMidPitch * sizeof(float4), a);
}

spx_status launch_fft_mid_chirp(spx_ctx* ctx, const FftPlan& plan, const float2* d_in, uint32_t beams,
                                uint32_t n_point, const float* d_win, uint32_t out_mode, float scale, void* d_out) {
  const FftPlan& sub = *plan.sub;
  const uint32_t m = plan.bm;
  void *scr = nullptr, *conv = nullptr;
  spx_status st = get_scratch(ctx, kSlotExchange, (size_t)beams * m * sizeof(float2), &scr);
  if (st == SPX_OK) st = get_scratch(ctx, kSlotChirp, (size_t)beams * m * sizeof(float2), &conv);
  if (st != SPX_OK) return st;
  const size_t smem = kMidRows * kMidPitch * sizeof(float4);
  MidRowsArgs a{};
  a.out = conv;
  a.chirp = plan.d_bfft;
  st = launch_mid(ctx, sub, d_in, beams, n_point, d_win, static_cast<float2*>(scr),
                  (const void*)mid_rows_kernel<kMidChirpMul>, smem, a, plan.d_chirp);
  if (st != SPX_OK) return st;
  a.out = d_out;
  a.out_mode = out_mode;
  a.scale = scale;
  a.chirp = plan.d_chirp;
  a.og = plan.g;
  const bool on_host = ctx->input_on_host;
  ctx->input_on_host = false;  // the convolution is in device memory
  st = launch_mid(ctx, sub, static_cast<const float2*>(conv), beams, m, nullptr, static_cast<float2*>(scr),
                  (const void*)mid_rows_kernel<kMidChirpPost>, smem, a);
  ctx->input_on_host = on_host;
  return st;
}

spx_status launch_fft_mid_rows(spx_ctx* ctx, const FftPlan& plan, const float2* d_in, uint32_t beams,
                               uint32_t n_point, const float* d_win, uint32_t klo, uint32_t khi, float2* d_rows) {
  MidRowsArgs a{};
  const uint32_t CB = 16 * plan.g.C;
  a.qlo = (klo / CB) & ~1u;  // whole pairs of elements
  a.qhi = khi > klo ? std::min<uint32_t>(kMidRow, (khi + CB - 1) / CB) : 0u;
  return launch_mid(ctx, plan, d_in, beams, n_point, d_win, d_rows, (const void*)mid_rows_window_kernel,
                    kMidRows * ps_len(kMidRow) * sizeof(float4), a);
}

}  // namespace spx
