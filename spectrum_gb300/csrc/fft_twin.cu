// fft_twin.cu — batched transforms of 2^a 3^b points, not a power of two: from
// 1024 to 8192 two beams per CTA in packed arithmetic, up to 16384 one.
//
// The odd strides of these plans leave no neighbours to pair inside a beam
// (fft_pair.cuh), so the two values of a pair are the same element of two beams:
// every twiddle, index and window value serves both, a 16-byte slot holds both,
// and the packed operations do the work of two scalar ones in one issue slot.
// The plan (CtPlan) and each beam's operations are those of fft_out_kernel, so
// the bits are too.  An odd last beam shares its CTA with itself.
//
// 2^25 points, fft_out_kernel<16> -> this: 1152 complex 197 -> 91 us, |X|^2 201 ->
// 87; 3072 inverse 204 -> 100; 4608 complex 229 -> 139; 6561 291 -> 197; 7776 281
// -> 200, {|X|, phase} 306 -> 263; about 340 beams 21 .. 24 -> 17 .. 19.  Bound by
// the one or two CTAs an SM holds above 4096 points (128 KB of slots and the
// register file), by issue below.  Pairing alone gave a tenth; the rest came with
// the layout of CtPlan's blocks, which needs no index computation per element.
#include <algorithm>

#include "fft_core.cuh"
#include "fft_pair.cuh"
#include "spx_internal.h"

namespace spx {

// Samples n0 + r step of both beams, windowed, zero beyond n_point (load_sample's
// products).
struct TwinSamples {
  const float2 *__restrict__ a, *__restrict__ b;
  uint32_t n_point;
  const float* __restrict__ win;
  template <int R>
  SPX_DEV void load(C2 (&v)[R], uint32_t n0, uint32_t step) const {
    float2 x[R], y[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t n = n0 + r * step;
      x[r] = y[r] = make_float2(0.f, 0.f);
      if (n < n_point) {
        x[r] = __ldcs(a + n);
        y[r] = __ldcs(b + n);
      }
    }
    if (win) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t n = n0 + r * step;
        if (n < n_point) {
          const float w = __ldg(win + n);
          x[r] = make_float2(__fmul_rn(x[r].x, w), __fmul_rn(x[r].y, w));
          y[r] = make_float2(__fmul_rn(y[r].x, w), __fmul_rn(y[r].y, w));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = C2{make_float2(x[r].x, y[r].x), make_float2(x[r].y, y[r].y)};
  }
};

// The slots between pass P - 1 and pass P lie in CtPlan's blocks: blocks of ns(P)
// elements, one unused slot (CtPlan::pad) after each behind a first pass of even
// radix, whose outputs would else meet in one bank.
SPX_DEV void twin_put(float4* s, C2 z) { *s = make_float4(z.x.x, z.x.y, z.y.x, z.y.y); }

// ct_first, ct_pass and ct_last_pass_out on pairs.
template <int M>
SPX_DEV void twin_first(float4* s, const TwinSamples& load, uint32_t tid) {
  using P = CtPlan<M>;
  constexpr int R = P::radix(0), B = M / R, T = P::T, Q = (B + T - 1) / T;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint32_t j = tid + q * T;
    if (B % T == 0 || q + 1 < Q || j < (uint32_t)B) {
      C2 v[R];
      load.load(v, j, B);
      PDft<R>::run(v);
#pragma unroll
      for (int r = 0; r < R; ++r) twin_put(s + j * (R + P::pad(1)) + r, v[r]);
    }
  }
  __syncthreads();
}
template <int M, int P, typename Out>
SPX_DEV void twin_pass(float4* s, const float2* __restrict__ tw, uint32_t tid, const Out& out) {
  using PL = CtPlan<M>;
  constexpr int R = PL::radix(P), Ns = PL::ns(P), B = M / R, T = PL::T, Q = (B + T - 1) / T;
  constexpr bool last = P + 1 == PL::npass;
  C2 v[Q][R];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint32_t j = tid + q * T;
    if (B % T == 0 || q + 1 < Q || j < (uint32_t)B) {
      const float4* p = s + j + PL::pad(P) * (j / Ns);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 z = p[r * (B + PL::pad(P) * (B / Ns))];
        v[q][r] = C2{make_float2(z.x, z.y), make_float2(z.z, z.w)};
      }
    }
  }
  if constexpr (!last) __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint32_t j = tid + q * T;
    if (B % T == 0 || q + 1 < Q || j < (uint32_t)B) {
      const uint32_t k = j % Ns;
      const float2* t = tw + PL::twoff(P) + k;
      if constexpr (R == 4) {
        const float2 w1 = tw4(tw + PL::twoff(P), k, Ns), w2 = cmul(w1, w1), w3 = cmul(w2, w1);
        v[q][1] = c2mul(v[q][1], C2{pk(w1.x), pk(w1.y)});
        v[q][2] = c2mul(v[q][2], C2{pk(w2.x), pk(w2.y)});
        v[q][3] = c2mul(v[q][3], C2{pk(w3.x), pk(w3.y)});
      } else {
#pragma unroll
        for (int r = 1; r < R; ++r) v[q][r] = c2mul(v[q][r], tw_both(t + (r - 1) * Ns));
      }
      PDft<R>::run(v[q]);
      float4* d = s + (j - k) * R + k + PL::pad(P + 1) * (j / Ns);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if constexpr (last)
          out(j + r * B, v[q][r]);
        else
          twin_put(d + r * Ns, v[q][r]);
      }
    }
  }
  if constexpr (!last) {
    __syncthreads();
    twin_pass<M, P + 1>(s, tw, tid, out);
  }
}

template <int M>
__global__ void __launch_bounds__(CtPlan<M>::T, 576 / CtPlan<M>::T)
fft_twin_kernel(const float2* __restrict__ in, uint32_t n_point, const float* __restrict__ win, FftGeom g,
                const float2* __restrict__ tw, void* __restrict__ out, uint32_t out_mode, float scale) {
  extern __shared__ float4 s4[];
  constexpr uint32_t T = CtPlan<M>::T;
  const uint32_t tid = threadIdx.x, b0 = 2 * blockIdx.x, b1 = min(b0 + 1, g.beams - 1);
  if (g.ahead && b0 + 2 * g.ahead < g.beams) {  // both beams (contiguous) of the CTA one residency wave later
    const uint32_t f = b0 + 2 * g.ahead, n = min(2u, g.beams - f);
    prefetch_l2(in + (size_t)f * n_point, (size_t)n * n_point * sizeof(float2), tid, T);
  }
  const TwinSamples ld{in + (size_t)b0 * n_point, in + (size_t)b1 * n_point, n_point, win};
  twin_first<M>(s4, ld, tid);
  if (out_mode == SPX_OUT_COMPLEX || out_mode == kOutComplexReversed) {
    const bool rev = out_mode == kOutComplexReversed;
    float2* o = reinterpret_cast<float2*>(out) + (size_t)b0 * M;
    twin_pass<M, 1>(s4, tw, tid, [&](uint32_t k, C2 z) {
      const uint32_t i = rev ? (k == 0 ? 0u : M - k) : k;
      if (rev) z = C2{pmul(z.x, pk(scale)), pmul(z.y, pk(scale))};
      o[i] = first_of(z);
      if (b1 != b0) o[M + i] = second_of(z);
    });
    return;
  }
  if (out_mode == SPX_OUT_MAG || out_mode == SPX_OUT_MAG2) {
    const bool squared = out_mode == SPX_OUT_MAG2;
    float* o = reinterpret_cast<float*>(out) + (size_t)b0 * M;
    twin_pass<M, 1>(s4, tw, tid, [&](uint32_t k, C2 z) {
      float m = mag2_rn(first_of(z)), n = mag2_rn(second_of(z));
      if (!squared) {
        m = __fsqrt_rn(m);
        n = __fsqrt_rn(n);
      }
      o[k] = __fmul_rn(m, scale);
      if (b1 != b0) o[M + k] = __fmul_rn(n, scale);
    });
    return;
  }
  // the other modes: from shared memory, one bin at a time (the last pass writes
  // the elements it read, in natural order)
  static_assert(CtPlan<M>::npass > 2, "no padding before the last pass");
  twin_pass<M, 1>(s4, tw, tid, [&](uint32_t k, C2 z) { twin_put(s4 + k, z); });
  __syncthreads();
#pragma unroll 4
  for (uint32_t k = tid; k < (uint32_t)M; k += T) {
    const float4 z = s4[k];
    store_bin(out, out_mode, scale, g, b0, k, make_float2(z.x, z.z));
    if (b1 != b0) store_bin(out, out_mode, scale, g, b1, k, make_float2(z.y, z.w));
  }
}

// 8748 .. 15552 points: pairs of beams would not fit the register file, so one
// beam per CTA in scalar arithmetic, at the compile-time plan (fft_core.cuh),
// where fft_out_kernel runs the passes with run-time radices and strides.  2^25
// points, complex: 8748 398 -> 290 us, 9216 301 -> 216, 12288 285 -> 205, 15552 313
// -> 237; inverse 286 -> 213 at 12288.
template <int M>
__global__ void __launch_bounds__(CtPlan<M>::T)
fft_solo_kernel(const float2* __restrict__ in, uint32_t n_point, const float* __restrict__ win, FftGeom g,
                const float2* __restrict__ tw, void* __restrict__ out, uint32_t out_mode, float scale) {
  extern __shared__ float2 s2[];
  const uint32_t tid = threadIdx.x, beam = blockIdx.x;
  prefetch_future_beam(g, in, n_point, beam, 0, tid, CtPlan<M>::T);
  const SampleLoader ld{in + (size_t)beam * n_point, n_point, win};
  if (out_mode == SPX_OUT_COMPLEX) {
    float2* o = reinterpret_cast<float2*>(out) + (size_t)beam * M;
    ct_local_fft_out<M>(s2, ld, tw, tid, [=](uint32_t k, float2 z) { o[k] = z; });
  } else {
    ct_local_fft_out<M>(s2, ld, tw, tid, BinOut{out, out_mode, scale, &g, beam});
  }
}

template <int M>
static const void* twin_kernel(uint32_t m) {
  if (m != M) return nullptr;
  if constexpr (M > 8192) return (const void*)fft_solo_kernel<M>;
  else return (const void*)fft_twin_kernel<M>;
}
static const void* twin_kernel_of(uint32_t m) {
  const void* k = nullptr;
  auto any = [&](auto... sizes) { ((k = k ? k : twin_kernel<decltype(sizes)::value>(m)), ...); };
#define SPX_TWIN(n) std::integral_constant<int, n>()
  any(SPX_TWIN(1152), SPX_TWIN(1296), SPX_TWIN(1458), SPX_TWIN(1536), SPX_TWIN(1728), SPX_TWIN(1944), SPX_TWIN(2187),
      SPX_TWIN(2304), SPX_TWIN(2592), SPX_TWIN(2916), SPX_TWIN(3072), SPX_TWIN(3456), SPX_TWIN(3888), SPX_TWIN(4374),
      SPX_TWIN(4608), SPX_TWIN(5184), SPX_TWIN(5832), SPX_TWIN(6144), SPX_TWIN(6561), SPX_TWIN(6912), SPX_TWIN(7776),
      SPX_TWIN(8748), SPX_TWIN(9216), SPX_TWIN(10368), SPX_TWIN(11664), SPX_TWIN(12288), SPX_TWIN(13122),
      SPX_TWIN(13824), SPX_TWIN(15552));
#undef SPX_TWIN
  return k;
}

bool twin_supported(const FftGeom& g) { return g.C == 1 && g.ept == 16 && twin_kernel_of(g.M) != nullptr; }

cudaError_t launch_fft_twin(const FftPlan& plan, const float2* d_in, uint32_t beams, uint32_t n_point,
                            const float* d_win, uint32_t out_mode, float scale, void* d_out, cudaStream_t stream,
                            bool prefetch) {
  FftGeom g = plan.g;
  const void* kfn = twin_kernel_of(g.M);
  const uint32_t threads = ((g.M + 15) / 16 + 31) / 32 * 32;
  const uint32_t per_cta = g.M > 8192 ? 1 : 2;
  const size_t smem = per_cta == 1 ? (size_t)sw_len(g.M) * sizeof(float2)
                                   : (size_t)(g.M + (g.radix[0] % 2 == 0 ? g.M / g.radix[0] : 0)) * sizeof(float4);
  cudaError_t e = configure_kernel(kfn, smem);
  if (e != cudaSuccess) return e;
  g.beams = beams;
  g.ahead = prefetch ? resident_ctas(kfn, threads, smem, 1) : 0u;
  void* args[] = {(void*)&d_in, (void*)&n_point, (void*)&d_win, (void*)&g,
                  (void*)&plan.d_tw_local, (void*)&d_out, (void*)&out_mode, (void*)&scale};
  return cudaLaunchKernel(kfn, dim3((beams + per_cta - 1) / per_cta), dim3(threads), args, smem, stream);
}

}  // namespace spx
