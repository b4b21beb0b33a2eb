// mlp.cu — learned sub-bin refinement of spectral peaks.
//
// No reference counterpart: the reference refines a peak with a 3-point
// parabola on |X| (include/spectrum/kernels/fft_kernel_sources_rocm.hpp:228-239),
// which for a Hann window is biased by up to a few hundredths of a bin
// (scalloping).  Here a small network learns the offset and the amplitude
// correction from the 5 bins around the peak.
//
// Network: 10 -> 64 -> 64 -> 2, GELU (erf form) after both hidden layers.
//   input : |X[k+d]| / |X[k]|                                   d = -2..2
//           wrap(arg(X[k+d] conj X[k]) + pi d (n_point-1)/nfft)  d = -2..2
//           (the linear phase of a symmetric window starting at sample 0 is
//            removed, so main-lobe phases sit near 0 and do not wrap)
//   output: y0 = offset of the tone from bin k, in bins
//           y1 = log(tone amplitude / |X[k]|)
// Weights: FP32 masters (Adam) and a BF16 copy; every product reads the BF16
// weights and accumulates in FP32; biases stay FP32.
// Training data comes from the library's own FFT: single-tone frames, features
// from the frame's nfft-point Hann spectrum, labels from a 16x zero-padded FFT
// of the same windowed frame (peak on the fine grid + 3-point parabola there).
// Inference keeps the parabolic result whenever the network's offset leaves
// the bin (|y0| > 0.5) or is not finite.
//
// Parameter layout (floats): W1[64][10] b1[64] W2[64][64] b2[64] W3[2][64] b3[2].
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

#include "mlp_device.cuh"
#include "spx_device.cuh"
#include "spx_internal.h"

namespace spx {

SPX_DEV float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) +
         z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// ---- training: forward, backward and the weight gradients of a tile in one CTA ----
// A CTA takes tiles of kTile rows and keeps everything between the layers in
// shared memory: activations as [unit][row] (pitch kTp: consecutive units or
// four-row quads of consecutive lanes hit different banks), the weights as FP32.
// Every product is a register tile fed by 128-bit shared loads.  The weight
// gradients stay in registers over the CTA's tiles and leave as one partial sum
// per CTA, added by mlp_reduce_kernel in CTA order: tiles are dealt to a number
// of CTAs that depends on the rows alone, so the gradient is the same bits on
// every run (no atomics).
// Bound: 28 kFLOP a row are a few microseconds of the FP32 pipe; the tile's
// chain of layers (seven barriers) and two launches are what is left.  One
// thread per output and layer took twelve launches with chains of 512 rows in as
// few as 16 CTAs: loss and gradients of 4096 rows 262 -> 21 us a call, error against
// FP64 1.3 .. 1.9e-7 -> 0.6e-7 (2^20 rows 1.22 ms).
constexpr int kTile = 32, kTp = kTile + 4;  // rows per tile; row pitch of [unit][row] arrays
constexpr int kWp = kH + 4;                 // row pitch of W2
constexpr int kW1p = 12;                    // row pitch of W1
constexpr uint32_t kMaxTileCtas = 304;      // two per SM
constexpr uint32_t kChain = 16;             // tiles (512 rows) added up in one FP32 chain
constexpr uint32_t kPart = kNParams + 2;    // floats of a partial sum: gradients, loss, padding

struct TileSmem {
  float w2[kH * kWp], w1[kH * kW1p], w3[kOut * kH], b1[kH], b2[kH], b3[kOut + 2];
  float x[kIn * kTp], h1[kH * kTp], h2[kH * kTp];
  float g1[kH * kTp], g2[kH * kTp];  // GELU' of layers 1, 2, then their dZ
  float dy[kOut * kTp];
};

struct TileArgs {
  const __nv_bfloat16* pb;
  const float* p;
  const float *x, *t;
  const uint32_t* mask;  // may be null
  uint32_t rows;
  // row j of the pass is row (pa (first + j) + pc) mod n of x, t and mask (an
  // affine permutation of [0, n), n a power of two), or row j when n = 0
  uint32_t n, first, pa, pc;
  float* y;     // forward: [rows][2]
  float* part;  // gradients: [CTAs][kPart]
};

SPX_DEV float dot4(float4 a, float4 b, float acc) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
SPX_DEV void fma4(float (&acc)[4], float w, float4 v) {
  acc[0] = fmaf(v.x, w, acc[0]);
  acc[1] = fmaf(v.y, w, acc[1]);
  acc[2] = fmaf(v.z, w, acc[2]);
  acc[3] = fmaf(v.w, w, acc[3]);
}

template <bool GRAD>
__global__ void __launch_bounds__(256)
mlp_tile_kernel(TileArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileSmem& s = *reinterpret_cast<TileSmem*>(smem_raw);
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < kH * kH; i += 256) s.w2[(i / kH) * kWp + i % kH] = __bfloat162float(a.pb[kOffW2 + i]);
  for (uint32_t i = tid; i < kH * kIn; i += 256) s.w1[(i / kIn) * kW1p + i % kIn] = __bfloat162float(a.pb[kOffW1 + i]);
  if (tid < kOut * kH) s.w3[tid] = __bfloat162float(a.pb[kOffW3 + tid]);
  if (tid < kH) {
    s.b1[tid] = a.p[kOffB1 + tid];
    s.b2[tid] = a.p[kOffB2 + tid];
  }
  if (tid < kOut) s.b3[tid] = a.p[kOffB3 + tid];
  auto source = [&](uint32_t j) { return a.n ? (a.pa * (a.first + j) + a.pc) & (a.n - 1) : j; };
  auto f4 = [](const float* p) { return *reinterpret_cast<const float4*>(p); };
  const uint32_t r4 = 4 * (tid & 7), up = tid >> 3;  // four rows, two units of the layers
  const uint32_t to = tid & 15, ti = tid >> 4;       // W2 gradient: units to + 16 j, inputs ti + 16 k
  // sums of up to kChain tiles, and of those sums
  float gw2[4][4] = {}, gw1[3] = {}, gw3 = 0.f, sw2[4][4] = {}, sw1[3] = {}, sw3 = 0.f, loss = 0.f;
  uint32_t chain = 0;
  const uint32_t tiles = (a.rows + kTile - 1) / kTile;
#pragma unroll 1
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t j0 = tile * kTile;
    for (uint32_t i = tid; i < kTile * kIn; i += 256) {
      const uint32_t r = i / kIn, c = i - r * kIn;
      s.x[c * kTp + r] = j0 + r < a.rows ? a.x[(size_t)source(j0 + r) * kIn + c] : 0.f;
    }
    __syncthreads();
    // layer 1, units up and up + 32
#pragma unroll
    for (uint32_t u = up; u < kH; u += 32) {
      float z[4] = {s.b1[u], s.b1[u], s.b1[u], s.b1[u]};
#pragma unroll
      for (uint32_t i = 0; i < kIn; ++i) fma4(z, s.w1[u * kW1p + i], f4(s.x + i * kTp + r4));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s.h1[u * kTp + r4 + q] = gelu(z[q]);
        if (GRAD) s.g1[u * kTp + r4 + q] = gelu_grad(z[q]);
      }
    }
    __syncthreads();
    // layer 2
    {
      float z[2][4];
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int q = 0; q < 4; ++q) z[e][q] = s.b2[up + 32 * e];
#pragma unroll 4
      for (uint32_t i = 0; i < kH; i += 4) {
        const float4 w0 = f4(s.w2 + up * kWp + i), w1 = f4(s.w2 + (up + 32) * kWp + i);
        const float4 h0 = f4(s.h1 + i * kTp + r4), h1 = f4(s.h1 + (i + 1) * kTp + r4),
                     h2 = f4(s.h1 + (i + 2) * kTp + r4), h3 = f4(s.h1 + (i + 3) * kTp + r4);
        fma4(z[0], w0.x, h0); fma4(z[0], w0.y, h1); fma4(z[0], w0.z, h2); fma4(z[0], w0.w, h3);
        fma4(z[1], w1.x, h0); fma4(z[1], w1.y, h1); fma4(z[1], w1.z, h2); fma4(z[1], w1.w, h3);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t at = (up + 32 * e) * kTp + r4 + q;
          s.h2[at] = gelu(z[e][q]);
          if (GRAD) s.g2[at] = gelu_grad(z[e][q]);
        }
    }
    __syncthreads();
    // layer 3: thread (row, output); masked mean squared error and its gradient
    if (tid < kTile * kOut) {
      const uint32_t r = tid & (kTile - 1), o = tid / kTile, j = j0 + r;
      float y = s.b3[o];
#pragma unroll 16
      for (uint32_t i = 0; i < kH; ++i) y = fmaf(s.h2[i * kTp + r], s.w3[o * kH + i], y);
      if constexpr (GRAD) {
        float d = 0.f;
        if (j < a.rows) {
          const uint32_t src = source(j);
          if (!a.mask || a.mask[src] != 0) d = y - a.t[(size_t)src * kOut + o];
        }
        const float n = (float)((uint64_t)a.rows * kOut);
        s.dy[o * kTp + r] = d * (2.0f / n);
        loss += d * d / n;
      } else if (j < a.rows) {
        a.y[(size_t)j * kOut + o] = y;
      }
    }
    if constexpr (GRAD) {
      __syncthreads();
      // dZ2 = (dY W3) GELU'(Z2), over g2
#pragma unroll
      for (uint32_t u = up; u < kH; u += 32) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        fma4(d, s.w3[u], f4(s.dy + r4));
        fma4(d, s.w3[kH + u], f4(s.dy + kTp + r4));
#pragma unroll
        for (int q = 0; q < 4; ++q) s.g2[u * kTp + r4 + q] *= d[q];
      }
      __syncthreads();
      // W3 and the biases of layers 2 and 3
      if (tid < kOut * kH) {
        const uint32_t o = tid / kH, i = tid % kH;
#pragma unroll
        for (int r = 0; r < kTile; r += 4) gw3 = dot4(f4(s.dy + o * kTp + r), f4(s.h2 + i * kTp + r), gw3);
      } else if (tid < kOut * kH + kH + kOut) {
        const uint32_t u = tid - kOut * kH;
        const float* d = u < kH ? s.g2 + u * kTp : s.dy + (u - kH) * kTp;
#pragma unroll
        for (int r = 0; r < kTile; r += 4) gw3 = dot4(f4(d + r), make_float4(1.f, 1.f, 1.f, 1.f), gw3);
      }
      // dZ1 = (dZ2 W2) GELU'(Z1), inputs 2 up and 2 up + 1, over g1
      {
        float d[2][4] = {};
#pragma unroll 8
        for (uint32_t o = 0; o < kH; ++o) {
          const float2 w = *reinterpret_cast<const float2*>(s.w2 + o * kWp + 2 * up);
          const float4 z = f4(s.g2 + o * kTp + r4);
          fma4(d[0], w.x, z);
          fma4(d[1], w.y, z);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int q = 0; q < 4; ++q) s.g1[(2 * up + e) * kTp + r4 + q] *= d[e][q];
      }
      // W2
#pragma unroll 2
      for (int r = 0; r < kTile; r += 4) {
        float4 z[4], h[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          z[k] = f4(s.g2 + (to + 16 * k) * kTp + r);
          h[k] = f4(s.h1 + (ti + 16 * k) * kTp + r);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) gw2[j][k] = dot4(z[j], h[k], gw2[j][k]);
      }
      __syncthreads();
      // W1 and its bias (input kIn)
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const uint32_t i = (tid + 256 * e) / kH, o = tid % kH;
        if (i > (uint32_t)kIn) break;
#pragma unroll
        for (int r = 0; r < kTile; r += 4)
          gw1[e] = dot4(f4(s.g1 + o * kTp + r), i < (uint32_t)kIn ? f4(s.x + i * kTp + r) : make_float4(1.f, 1.f, 1.f, 1.f),
                        gw1[e]);
      }
      if (++chain == kChain) {
        chain = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            sw2[j][k] += gw2[j][k];
            gw2[j][k] = 0.f;
          }
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          sw1[e] += gw1[e];
          gw1[e] = 0.f;
        }
        sw3 += gw3;
        gw3 = 0.f;
      }
    }
    __syncthreads();  // the tile's arrays are rewritten by the next one
  }
  if constexpr (GRAD) {
    float* g = a.part + (size_t)blockIdx.x * kPart;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) g[kOffW2 + (to + 16 * j) * kH + ti + 16 * k] = sw2[j][k] + gw2[j][k];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const uint32_t i = (tid + 256 * e) / kH, o = tid % kH;
      if (i < (uint32_t)kIn) g[kOffW1 + o * kIn + i] = sw1[e] + gw1[e];
      if (i == (uint32_t)kIn) g[kOffB1 + o] = sw1[e] + gw1[e];
    }
    gw3 += sw3;
    if (tid < kOut * kH) g[kOffW3 + tid] = gw3;
    else if (tid < kOut * kH + kH) g[kOffB2 + tid - kOut * kH] = gw3;
    else if (tid < kOut * kH + kH + kOut) g[kOffB3 + tid - kOut * kH - kH] = gw3;
    if (tid < kTile * kOut) {  // two warps
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
      if ((tid & 31) == 0) s.dy[tid >> 5] = loss;
    }
    __syncthreads();
    if (tid == 0) g[kNParams] = s.dy[0] + s.dy[1];
  }
}

// Parameter i's place in the staged weights (MlpWeights: the layers' matrices as
// FP32 of their BF16 rounding, the hidden ones transposed), and its value there.
SPX_DEV void stage_param(MlpWeights* w, uint32_t i, float p, __nv_bfloat16 pb) {
  const float v = __bfloat162float(pb);
  if (i < kOffB1) w->w1t[(i % kIn) * kH + i / kIn] = v;
  else if (i < kOffW2) w->b1[i - kOffB1] = p;
  else if (i < kOffB2) w->w2t[((i - kOffW2) % kH) * kH + (i - kOffW2) / kH] = v;
  else if (i < kOffW3) w->b2[i - kOffB2] = p;
  else if (i < kOffB3) w->w3[i - kOffW3] = v;
  else w->b3[i - kOffB3] = p;
}

// The partial sums of `parts` CTAs added in a fixed order: 32 parameters per
// CTA, eight threads each.  The last "parameter" is the loss (added to *loss).
// grad != null takes the gradient; else one Adam step of the FP32 masters
// (bias-corrected) and the BF16 copy.
struct AdamArgs {
  float *p, *m, *v;
  __nv_bfloat16* pb;
  MlpWeights* staged;
  float lr, b1, b2, eps, c1, c2;
};
__global__ void __launch_bounds__(256)
mlp_reduce_kernel(const float* __restrict__ part, uint32_t parts, float* __restrict__ grad, float* __restrict__ loss,
                  AdamArgs ad) {
  __shared__ float sum[8][32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (i <= (uint32_t)kNParams)
    for (uint32_t c = w; c < parts; c += 8) acc += part[(size_t)c * kPart + i];
  sum[w][lane] = acc;
  __syncthreads();
  if (w != 0 || i > (uint32_t)kNParams) return;
  float g = sum[0][lane];
#pragma unroll
  for (int k = 1; k < 8; ++k) g += sum[k][lane];
  if (i == (uint32_t)kNParams) {
    if (loss) *loss += g;
    return;
  }
  if (grad) {
    grad[i] = g;
    return;
  }
  const float mi = ad.b1 * ad.m[i] + (1.f - ad.b1) * g;
  const float vi = ad.b2 * ad.v[i] + (1.f - ad.b2) * g * g;
  ad.m[i] = mi;
  ad.v[i] = vi;
  const float pi = ad.p[i] - ad.lr * (mi / ad.c1) / (sqrtf(vi / ad.c2) + ad.eps);
  ad.p[i] = pi;
  const __nv_bfloat16 b = __float2bfloat16_rn(pi);
  ad.pb[i] = b;
  stage_param(ad.staged, i, pi, b);
}

__global__ void to_bf16_kernel(const float* __restrict__ p, __nv_bfloat16* __restrict__ pb, MlpWeights* __restrict__ w,
                               uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const __nv_bfloat16 b = __float2bfloat16_rn(p[i]);
  pb[i] = b;
  stage_param(w, i, p[i], b);
}

// ---- features -------------------------------------------------------------------
// Features of the peak at bin k of a spectrum in device memory (needs bins
// k-2..k+2); false at the edges or when |X[k]| is 0.
struct GlobalBins {
  const float2* f;
  SPX_DEV float2 operator()(uint32_t k) const { return f[k]; }
};
SPX_DEV bool peak_features(const float2* f, uint32_t n_point, uint32_t nfft, uint32_t k, float* feat) {
  return peak_features_at(GlobalBins{f}, n_point, nfft, k, feat);
}

// ---- training data ----------------------------------------------------------------
SPX_DEV uint64_t mix64(uint64_t z) {  // splitmix64 finaliser
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
SPX_DEV float u01(uint64_t key) { return (float)(mix64(key) >> 40) * (1.0f / 16777216.0f); }
SPX_DEV float gauss(uint64_t key) {  // Box-Muller, one of the pair
  const float u1 = fmaxf(u01(key), 1e-7f), u2 = u01(key ^ 0xA5A5A5A5A5A5A5A5ull);
  return sqrtf(-2.f * logf(u1)) * cospif(2.f * u2);
}

// One single-tone frame per block: x[t] = exp(i(2 pi f t + phi)) + sigma (n_re + i n_im),
// f ~ U[fmin, fmax) cycles/sample, phi ~ U[0, 2 pi), SNR ~ U[snr_lo, snr_hi] dB
// (sigma = 10^(-SNR/20), total complex noise power sigma^2).
__global__ void gen_frames_kernel(uint64_t seed, uint32_t frame0, uint32_t n, float fmin,
                                  float fmax, float snr_lo, float snr_hi, float2* __restrict__ x,
                                  float* __restrict__ truth) {
  const uint32_t fr = blockIdx.x;
  const uint64_t key = mix64(seed ^ mix64(frame0 + fr));
  const float f = fmin + (fmax - fmin) * u01(key ^ 1);
  const float ph = u01(key ^ 2);  // cycles
  const float snr = snr_lo + (snr_hi - snr_lo) * u01(key ^ 3);
  const float s = powf(10.f, -snr / 20.f) * 0.70710678118654752f;
  if (threadIdx.x == 0 && truth) {
    truth[(size_t)fr * 2] = f;
    truth[(size_t)fr * 2 + 1] = snr;
  }
  for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) {
    const double cyc = (double)f * (double)t + (double)ph;
    const float frac = (float)(cyc - floor(cyc));
    float sn, cs;
    sincospif(2.f * frac, &sn, &cs);
    const uint64_t nk = mix64(key + t);
    x[(size_t)fr * n + t] = make_float2(cs + s * gauss(nk), sn + s * gauss(nk ^ 0x5851F42D4C957F2Dull));
  }
}

// Per frame: k = argmax |X| over [2, nfft/2 - 2) (largest value, lowest bin);
// features at k; labels from the 16x zero-padded spectrum X16 (fine-grid peak
// within +-24 fine bins of 16 k, then a 3-point parabola on the fine grid):
// target = (fine offset, log(fine amplitude / |X[k]|)); parabolic = (k, the
// 3-point coarse parabola offset: the method without the network); valid = 0
// for unusable frames.
__global__ void frame_labels_kernel(const float2* __restrict__ X, const float2* __restrict__ X16,
                                    uint32_t nfft, float* __restrict__ feat, float* __restrict__ tgt,
                                    float* __restrict__ par, uint32_t* __restrict__ valid) {
  const uint32_t fr = blockIdx.x;
  const float2* f = X + (size_t)fr * nfft;
  const float2* g = X16 + (size_t)fr * nfft * 16;
  __shared__ uint64_t best[32];
  uint64_t key = 0;
  for (uint32_t k = 2 + threadIdx.x; k + 2 < nfft / 2; k += blockDim.x) {
    const uint64_t kk = ((uint64_t)__float_as_uint(mag_rn(f[k])) << 32) | (uint32_t)(~k);
    key = kk > key ? kk : key;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const uint64_t w = __shfl_xor_sync(0xffffffffu, key, o);
    key = w > key ? w : key;
  }
  if ((threadIdx.x & 31) == 0) best[threadIdx.x >> 5] = key;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (uint32_t w = 1; w < blockDim.x / 32; ++w) key = best[w] > key ? best[w] : key;
  const uint32_t k = ~(uint32_t)key;
  float fe[kIn];
  bool ok = key != 0 && peak_features(f, nfft, nfft, k, fe);
  float off = 0.f, la = 0.f, pd = 0.f;
  if (ok) {
    uint32_t mbest = 16 * k;
    float vbest = -1.f;
    for (int d = -24; d <= 24; ++d) {
      const uint32_t m = 16 * k + d;
      const float v = mag_rn(g[m]);
      if (v > vbest) { vbest = v; mbest = m; }
    }
    const float yl = mag_rn(g[mbest - 1]), yc = vbest, yr = mag_rn(g[mbest + 1]);
    const float den = yl - 2.f * yc + yr;
    const float dfine = fabsf(den) > 1e-20f ? fminf(fmaxf(0.5f * (yl - yr) / den, -0.5f), 0.5f) : 0.f;
    const float amp = yc - 0.25f * (yl - yr) * dfine;
    const float mc = mag_rn(f[k]);
    off = ((float)mbest - 16.f * (float)k + dfine) * (1.f / 16.f);
    la = logf(amp / mc);
    ok = amp > 0.f && fabsf(off) < 1.0f && isfinite(la);
    const float cl = mag_rn(f[k - 1]), cr = mag_rn(f[k + 1]);
    const float cden = cl - 2.f * mc + cr;
    pd = fabsf(cden) > 1e-10f ? fminf(fmaxf(0.5f * (cl - cr) / cden, -0.5f), 0.5f) : 0.f;
  }
  for (int i = 0; i < kIn; ++i) feat[(size_t)fr * kIn + i] = ok ? fe[i] : 0.f;
  tgt[(size_t)fr * 2] = ok ? off : 0.f;
  tgt[(size_t)fr * 2 + 1] = ok ? la : 0.f;
  par[(size_t)fr * 2] = (float)k;
  par[(size_t)fr * 2 + 1] = pd;
  valid[fr] = ok ? 1u : 0u;
}

// ---- inference: one warp per peak ------------------------------------------------
// mlp_forward_warp (mlp_device.cuh): lane l owns hidden units l and l + 32 of
// both layers; the layer-1 outputs go through a per-warp shared row; the 2
// outputs are warp sums.  Weights are staged once per block in shared memory
// (BF16 values widened to FP32, exact).
constexpr int kRefineWarps = 8;
struct RefineSmem {
  MlpWeights w;
  float h[kRefineWarps][kH];
  float x[kRefineWarps][kIn];
};

// Bins around the peak at bin k, kept as k - 2 .. k + 2.
struct CtxBins {
  const float2* c;
  uint32_t k;
  SPX_DEV float2 operator()(uint32_t b) const { return c[b + 2 - k]; }
};

// CTX: `fft` holds each peak's five bins instead of the spectra, and the launch
// may begin before the search that writes them has ended (its CTAs that find room
// beside the search's last wave stage the weights meanwhile).
template <bool CTX>
__global__ void __launch_bounds__(kRefineWarps * 32)
mlp_refine_kernel(const MlpWeights* __restrict__ staged, const float2* __restrict__ fft, uint32_t n_point,
                  uint32_t nfft, uint32_t beams, uint32_t K, float fs, MaxValueDev* __restrict__ peaks,
                  const uint32_t* __restrict__ counts, float* __restrict__ amp_out,
                  uint32_t* __restrict__ used_mlp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RefineSmem& s = *reinterpret_cast<RefineSmem*>(smem_raw);
  static_assert(sizeof(MlpWeights) % 8 == 0, "copied in pairs of floats");
  for (uint32_t i = threadIdx.x; i < sizeof(MlpWeights) / 8; i += blockDim.x)
    reinterpret_cast<float2*>(&s.w)[i] = __ldg(reinterpret_cast<const float2*>(staged) + i);
  if constexpr (CTX) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("" : "+l"(fft), "+l"(counts), "+l"(peaks)::"memory");  // nothing of them is read earlier
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t total = (uint64_t)beams * K;
  const uint64_t stride = (uint64_t)gridDim.x * kRefineWarps;
  for (uint64_t idx = (uint64_t)blockIdx.x * kRefineWarps + warp; idx < total; idx += stride) {
    const uint32_t beam = (uint32_t)(idx / K), j = (uint32_t)(idx % K);
    if (j >= counts[beam]) continue;  // warp-uniform
    MaxValueDev mv = peaks[idx];
    // the features, offset d = lane - 2 on lanes 0..4 (peak_features_at's
    // arithmetic, one offset per lane)
    const uint32_t k = mv.index;
    const auto bins = [&] {
      if constexpr (CTX) return CtxBins{fft + idx * 5, k};
      else return GlobalBins{fft + (size_t)beam * nfft};
    }();
    bool good = k >= 2 && k + 2 < nfft;
    float2 c = make_float2(0.f, 0.f);
    float mc = 0.f;
    if (good) {
      c = bins(k);
      mc = mag_rn(c);
      good = mc > 0.f;
    }
    if (good && lane < 5)
      peak_feature_pair(bins, c, mc, peak_lin(n_point, nfft), k, (int)lane - 2, &s.x[warp][lane], &s.x[warp][lane + 5]);
    __syncwarp();
    float y0 = 0.f, y1 = 0.f;
    if (good) mlp_forward_warp(s.w, s.x[warp], s.h[warp], lane, &y0, &y1);
    __syncwarp();
    if (lane == 0) {
      float amp;
      const bool use = mlp_apply(mv, good, y0, y1, fs, nfft, &amp);
      if (use) peaks[idx] = mv;
      if (amp_out) amp_out[idx] = amp;
      if (used_mlp) used_mlp[idx] = use ? 1u : 0u;
    }
  }
}

}  // namespace spx

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
using namespace spx;

struct spx_mlp {
  int device = 0;
  float* d_p = nullptr;           // FP32 masters
  float* d_m = nullptr;           // Adam first moment
  float* d_v = nullptr;           // Adam second moment
  __nv_bfloat16* d_pb = nullptr;  // BF16 copy read by every product
  MlpWeights* d_staged = nullptr; // the weights as the refine kernel stages them
  float* d_work = nullptr;        // partial sums of the gradients
  size_t work_floats = 0;
  uint64_t step = 0;              // Adam step count
};

namespace spx {
void mlp_device_params(const spx_mlp* mlp, const void** pb, const float** p, int* device) {
  *pb = mlp->d_pb;
  *p = mlp->d_p;
  *device = mlp->device;
}
}  // namespace spx

namespace {

unsigned nblocks(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// CTAs of a pass over `rows` rows (a number that depends on the rows alone).
uint32_t tile_ctas(uint32_t rows) { return std::min<uint32_t>((rows + kTile - 1) / kTile, kMaxTileCtas); }

// Room for the partial sums of a pass.
spx_status ensure_work(spx_ctx* ctx, spx_mlp* m, uint32_t rows) {
  const size_t need = (size_t)tile_ctas(rows) * kPart;
  if (m->work_floats < need) {
    cudaError_t e = cudaSuccess;
    if (m->d_work) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess && m->d_work) e = cudaFree(m->d_work);
    m->d_work = nullptr;
    m->work_floats = 0;
    if (e == cudaSuccess) e = cudaMalloc(&m->d_work, need * sizeof(float));
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc(mlp partial sums)");
    m->work_floats = need;
  }
  return SPX_OK;
}

template <bool GRAD>
spx_status launch_tiles(spx_ctx* ctx, const spx_mlp* m, TileArgs a) {
  a.pb = m->d_pb;
  a.p = m->d_p;
  a.part = m->d_work;
  const void* kfn = (const void*)mlp_tile_kernel<GRAD>;
  cudaError_t e = configure_kernel(kfn, sizeof(TileSmem));
  if (e != cudaSuccess) return cuda_fail(ctx, e, "configure mlp_tile_kernel");
  mlp_tile_kernel<GRAD><<<tile_ctas(a.rows), 256, sizeof(TileSmem), ctx->stream>>>(a);
  e = cudaGetLastError();
  return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, "launch mlp_tile_kernel");
}

// Loss and gradient of a pass; the gradient into d_grad, or (null) one Adam step.
spx_status backward(spx_ctx* ctx, spx_mlp* m, const TileArgs& a, float* d_loss, float* d_grad, float lr) {
  spx_status st = ensure_work(ctx, m, a.rows);
  if (st == SPX_OK) st = launch_tiles<true>(ctx, m, a);
  if (st != SPX_OK) return st;
  AdamArgs ad{};
  if (!d_grad) {
    m->step += 1;
    ad = AdamArgs{m->d_p, m->d_m, m->d_v, m->d_pb, m->d_staged, lr, 0.9f, 0.999f, 1e-8f,
                  1.f - (float)std::pow(0.9, (double)m->step), 1.f - (float)std::pow(0.999, (double)m->step)};
  }
  mlp_reduce_kernel<<<nblocks(kNParams + 1, 32), 256, 0, ctx->stream>>>(m->d_work, tile_ctas(a.rows), d_grad, d_loss, ad);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, "launch mlp_reduce_kernel");
}

spx_status launch_status(spx_ctx* ctx, const char* what) {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, what);
}

template <bool CTX>
spx_status launch_refine(spx_ctx* ctx, const spx_mlp* m, const float2* d_bins, uint32_t beams, uint32_t n_point,
                         uint32_t nfft, float fs, uint32_t K, spx_max_value* d_peaks, const uint32_t* d_counts,
                         float* d_amplitude, uint32_t* d_used) {
  const size_t smem = sizeof(RefineSmem);
  cudaError_t e = configure_kernel((const void*)mlp_refine_kernel<CTX>, smem);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "spx_mlp_refine: configure");
  const uint64_t warps = (uint64_t)beams * K;
  const unsigned grid = (unsigned)std::min<uint64_t>((warps + kRefineWarps - 1) / kRefineWarps,
                                                     (uint64_t)ctx->sm_count * 8);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kRefineWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute overlap[1];
  overlap[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = overlap;
  cfg.numAttrs = CTX ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, mlp_refine_kernel<CTX>, (const MlpWeights*)m->d_staged, d_bins, n_point, nfft, beams, K,
                         fs, reinterpret_cast<MaxValueDev*>(d_peaks), d_counts, d_amplitude, d_used);
  return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, "spx_mlp_refine");
}

}  // namespace

namespace spx {
spx_status launch_mlp_refine_ctx(spx_ctx* ctx, const spx_mlp* m, const float2* d_ctx, uint32_t beams,
                                 uint32_t n_point, uint32_t nfft, float fs, uint32_t K, spx_max_value* d_peaks,
                                 const uint32_t* d_counts, float* d_amplitude, uint32_t* d_used) {
  return launch_refine<true>(ctx, m, d_ctx, beams, n_point, nfft, fs, K, d_peaks, d_counts, d_amplitude, d_used);
}
}  // namespace spx

extern "C" {

uint32_t spx_mlp_param_count(void) { return kNParams; }

spx_status spx_mlp_create(spx_ctx* ctx, uint64_t seed, spx_mlp** out) {
  if (!ctx || !out) return SPX_ERR_INVALID_ARG;
  *out = nullptr;
  DeviceGuard guard(ctx->device);
  auto* m = new (std::nothrow) spx_mlp();
  if (!m) return fail(ctx, SPX_ERR_OUT_OF_MEMORY, "spx_mlp_create: host allocation failed");
  m->device = ctx->device;
  cudaError_t e = cudaSuccess;
  float** bufs[] = {&m->d_p, &m->d_m, &m->d_v};
  for (float** b : bufs)
    if (e == cudaSuccess) e = cudaMalloc(b, kNParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&m->d_pb, kNParams * sizeof(__nv_bfloat16));
  if (e == cudaSuccess) e = cudaMalloc(&m->d_staged, sizeof(MlpWeights));
  if (e != cudaSuccess) {
    spx_mlp_destroy(m);
    return cuda_fail(ctx, e, "cudaMalloc(mlp parameters)");
  }
  // Uniform (He-style) initialisation from a seeded 64-bit LCG; biases 0.
  std::vector<float> p(kNParams, 0.f);
  uint64_t st = seed;
  auto next = [&]() {
    st = st * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(st >> 11) * (2.0 / 9007199254740992.0) - 1.0;  // U[-1, 1)
  };
  for (int i = 0; i < kH * kIn; ++i) p[kOffW1 + i] = (float)(next() * std::sqrt(6.0 / kIn));
  for (int i = 0; i < kH * kH; ++i) p[kOffW2 + i] = (float)(next() * std::sqrt(6.0 / kH));
  for (int i = 0; i < kOut * kH; ++i) p[kOffW3 + i] = (float)(next() * std::sqrt(1.0 / kH));
  const spx_status s = spx_mlp_set_params(ctx, m, p.data());
  if (s != SPX_OK) {
    spx_mlp_destroy(m);
    return s;
  }
  *out = m;
  return SPX_OK;
}

spx_status spx_mlp_destroy(spx_mlp* m) {
  if (!m) return SPX_OK;
  DeviceGuard guard(m->device);
  cudaFree(m->d_p);
  cudaFree(m->d_m);
  cudaFree(m->d_v);
  cudaFree(m->d_pb);
  cudaFree(m->d_staged);
  cudaFree(m->d_work);
  delete m;
  return SPX_OK;
}

spx_status spx_mlp_set_params(spx_ctx* ctx, spx_mlp* m, const float* host_params) {
  if (!ctx || !m || !host_params) return SPX_ERR_INVALID_ARG;
  DeviceGuard guard(ctx->device);
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpy(m->d_p, host_params, kNParams * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(m->d_m, 0, kNParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(m->d_v, 0, kNParams * sizeof(float));
  if (e != cudaSuccess) return cuda_fail(ctx, e, "spx_mlp_set_params");
  to_bf16_kernel<<<nblocks(kNParams, 256), 256, 0, ctx->stream>>>(m->d_p, m->d_pb, m->d_staged, kNParams);
  m->step = 0;
  e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, "spx_mlp_set_params");
}

spx_status spx_mlp_get_params(spx_ctx* ctx, spx_mlp* m, float* host_params) {
  if (!ctx || !m || !host_params) return SPX_ERR_INVALID_ARG;
  DeviceGuard guard(ctx->device);
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpy(host_params, m->d_p, kNParams * sizeof(float), cudaMemcpyDeviceToHost);
  return e == cudaSuccess ? SPX_OK : cuda_fail(ctx, e, "spx_mlp_get_params");
}

spx_status spx_mlp_forward(spx_ctx* ctx, spx_mlp* m, const float* d_x, uint32_t rows, float* d_y) {
  if (!ctx || !m) return SPX_ERR_INVALID_ARG;
  if (rows == 0) return SPX_OK;
  if (!d_x || !d_y) return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_forward: null pointer");
  DeviceGuard guard(ctx->device);
  TileArgs a{};
  a.x = d_x;
  a.rows = rows;
  a.y = d_y;
  // an output over the input: through scratch (a CTA would write rows another still reads)
  const size_t y_bytes = (size_t)rows * kOut * sizeof(float);
  const uintptr_t x0 = reinterpret_cast<uintptr_t>(d_x), y0 = reinterpret_cast<uintptr_t>(d_y);
  if (y0 >= x0 + (size_t)rows * kIn * sizeof(float) || x0 >= y0 + y_bytes) return launch_tiles<false>(ctx, m, a);
  void* tmp = nullptr;
  spx_status st = get_scratch(ctx, kSlotWork, y_bytes, &tmp);
  if (st != SPX_OK) return st;
  a.y = static_cast<float*>(tmp);
  st = launch_tiles<false>(ctx, m, a);
  if (st != SPX_OK) return st;
  cudaMemcpyAsync(d_y, tmp, y_bytes, cudaMemcpyDeviceToDevice, ctx->stream);
  return launch_status(ctx, "spx_mlp_forward");
}

spx_status spx_mlp_gradients(spx_ctx* ctx, spx_mlp* m, const float* d_x, const float* d_t,
                             const uint32_t* d_mask, uint32_t rows, float* d_grad, float* d_loss) {
  if (!ctx || !m) return SPX_ERR_INVALID_ARG;
  if (!d_x || !d_t || !d_grad || rows == 0)
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_gradients: null pointer or no rows");
  DeviceGuard guard(ctx->device);
  TileArgs a{};
  a.x = d_x;
  a.t = d_t;
  a.mask = d_mask;
  a.rows = rows;
  return backward(ctx, m, a, d_loss, d_grad, 0.f);
}

spx_status spx_mlp_train_step(spx_ctx* ctx, spx_mlp* m, const float* d_x, const float* d_t,
                              const uint32_t* d_mask, uint32_t rows, float lr, float* d_loss) {
  if (!ctx || !m) return SPX_ERR_INVALID_ARG;
  if (!d_x || !d_t || rows == 0)
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_train_step: null pointer or no rows");
  if (!(lr > 0.f) || !std::isfinite(lr)) return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_train_step: lr must be > 0");
  DeviceGuard guard(ctx->device);
  TileArgs a{};
  a.x = d_x;
  a.t = d_t;
  a.mask = d_mask;
  a.rows = rows;
  return backward(ctx, m, a, d_loss, nullptr, lr);
}

spx_status spx_mlp_train(spx_ctx* ctx, spx_mlp* m, const float* d_feat, const float* d_target,
                         const uint32_t* d_valid, uint32_t rows, uint32_t batch, uint32_t epochs,
                         float lr_max, float lr_min, uint64_t seed, float* d_epoch_loss) {
  if (!ctx || !m) return SPX_ERR_INVALID_ARG;
  if (!d_feat || !d_target) return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_train: null pointer");
  if (rows == 0 || (rows & (rows - 1)) || batch == 0 || batch > rows)
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_train: rows must be a power of two >= batch > 0");
  if (!(lr_max > 0.f) || !(lr_min > 0.f) || lr_min > lr_max || !std::isfinite(lr_max))
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_train: need 0 < lr_min <= lr_max");
  DeviceGuard guard(ctx->device);
  spx_status st = SPX_OK;
  if (d_epoch_loss) cudaMemsetAsync(d_epoch_loss, 0, (size_t)epochs * sizeof(float), ctx->stream);
  const uint32_t steps_per_epoch = rows / batch;
  const double total = (double)steps_per_epoch * epochs;
  uint64_t rs = seed;
  auto next = [&]() {
    rs = rs * 6364136223846793005ull + 1442695040888963407ull;
    return (uint32_t)(rs >> 32);
  };
  uint64_t step = 0;
  for (uint32_t ep = 0; ep < epochs; ++ep) {
    const uint32_t pa = next() | 1u, pc = next();
    for (uint32_t s = 0; s < steps_per_epoch; ++s, ++step) {
      // cosine decay from lr_max to lr_min over the whole run
      const double cosv = 0.5 * (1.0 + std::cos(3.14159265358979323846 * (double)step / total));
      const float lr = (float)(lr_min + (lr_max - lr_min) * cosv);
      TileArgs t{};
      t.x = d_feat;
      t.t = d_target;
      t.mask = d_valid;
      t.rows = batch;
      t.n = rows;
      t.first = s * batch;
      t.pa = pa;
      t.pc = pc;
      st = backward(ctx, m, t, d_epoch_loss ? d_epoch_loss + ep : nullptr, nullptr, lr);
      if (st != SPX_OK) return st;
    }
  }
  // per-epoch loss: mean over the epoch's steps
  if (d_epoch_loss) {
    std::vector<float> h(epochs);
    cudaError_t e = cudaMemcpyAsync(h.data(), d_epoch_loss, epochs * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    for (auto& v : h) v /= (float)steps_per_epoch;
    if (e == cudaSuccess) e = cudaMemcpy(d_epoch_loss, h.data(), epochs * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "spx_mlp_train loss");
  }
  return SPX_OK;
}

spx_status spx_mlp_make_frames(spx_ctx* ctx, uint64_t seed, uint32_t frame0, uint32_t frames,
                               uint32_t nfft, float snr_lo_db, float snr_hi_db, float* d_feat,
                               float* d_target, float* d_parabolic, uint32_t* d_valid,
                               float* d_truth) {
  if (!ctx) return SPX_ERR_INVALID_ARG;
  if (frames == 0) return SPX_OK;
  if (!d_feat || !d_target || !d_parabolic || !d_valid)
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_make_frames: null pointer");
  if (nfft < 64 || nfft > 4096 || (nfft & (nfft - 1)))
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_make_frames: nfft must be a power of two in [64, 4096]");
  if (!(snr_lo_db <= snr_hi_db) || !std::isfinite(snr_lo_db) || !std::isfinite(snr_hi_db))
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_make_frames: need finite snr_lo_db <= snr_hi_db");
  DeviceGuard guard(ctx->device);
  // frames x, spectra X and 16x zero-padded judge spectra X16, chunk by chunk
  const uint32_t chunk = std::min<uint32_t>(frames, (1u << 24) / nfft);
  const size_t pts = (size_t)chunk * nfft;
  void* scr = nullptr;
  spx_status st = get_scratch(ctx, kSlotSpectrum, 18 * pts * sizeof(float2), &scr);
  if (st != SPX_OK) return st;
  float2* x = static_cast<float2*>(scr);
  float2* X = x + pts;
  float2* X16 = X + pts;
  const float fmin = 4.0f / nfft, fmax = 0.5f - 4.0f / nfft;
  for (uint32_t f0 = 0; f0 < frames; f0 += chunk) {
    const uint32_t n = std::min(chunk, frames - f0);
    gen_frames_kernel<<<n, 256, 0, ctx->stream>>>(seed, frame0 + f0, nfft, fmin, fmax, snr_lo_db, snr_hi_db, x,
                                                  d_truth ? d_truth + (size_t)f0 * 2 : nullptr);
    st = launch_status(ctx, "spx_mlp_make_frames");
    if (st != SPX_OK) return st;
    st = spx_fft(ctx, x, n, nfft, nfft, SPX_WINDOW_HANN, SPX_OUT_COMPLEX, 1.0f, X);
    if (st != SPX_OK) return st;
    st = spx_fft(ctx, x, n, nfft, nfft * 16, SPX_WINDOW_HANN, SPX_OUT_COMPLEX, 1.0f, X16);
    if (st != SPX_OK) return st;
    frame_labels_kernel<<<n, 256, 0, ctx->stream>>>(X, X16, nfft, d_feat + (size_t)f0 * kIn,
                                                    d_target + (size_t)f0 * 2, d_parabolic + (size_t)f0 * 2,
                                                    d_valid + f0);
    st = launch_status(ctx, "spx_mlp_make_frames");
    if (st != SPX_OK) return st;
  }
  return SPX_OK;
}

spx_status spx_mlp_refine(spx_ctx* ctx, spx_mlp* m, const void* d_fft, uint32_t beams,
                          uint32_t n_point, uint32_t nfft, float sample_rate, uint32_t K,
                          spx_max_value* d_peaks, const uint32_t* d_counts, float* d_amplitude,
                          uint32_t* d_used_mlp) {
  if (!ctx || !m) return SPX_ERR_INVALID_ARG;
  if ((uint64_t)beams * K == 0) return SPX_OK;
  if (!d_fft || !d_peaks || !d_counts) return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_refine: null pointer");
  if (nfft < 5 || n_point == 0 || n_point > nfft)
    return fail(ctx, SPX_ERR_INVALID_ARG, "spx_mlp_refine: need 5 <= nfft and 0 < n_point <= nfft");
  DeviceGuard guard(ctx->device);
  return launch_refine<false>(ctx, m, static_cast<const float2*>(d_fft), beams, n_point, nfft, sample_rate, K, d_peaks,
                              d_counts, d_amplitude, d_used_mlp);
}

}  // extern "C"
