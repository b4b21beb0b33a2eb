// batch_rows.cuh — the two transform launches of a batch's larger beams: every
// beam of C x M points, C >= 2, M one of the sizes of BrSizes, in items of a few
// thousand points.
//
// The plan is the context's (C-point cross stage, then the local radices
// R0, R1, ...), element for element the same operations, so the spectra are the
// bits of the cluster kernel; the data crosses device memory after the local
// FFT's first pass (as in fft_mid.cu) instead of before it:
//   launch 1: for the columns j of a tile, the C-point DFTs over n1 of the
//     windowed samples n = M n1 + L r + j (L = M / R0), times W_N^{n2 k1}, then
//     the R0-point DFTs over r;
//   launch 2: the passes R1, R2, ... act on each row (k1, r0) alone: an L-point
//     FFT over j in row coordinates whose twiddles depend on r0.
// Rows r0 = 2i, 2i + 1 of one k1 run as a pair in packed arithmetic
// (fft_pair.cuh): one value of each row in a register pair, so any radix and any
// odd stride will do.  A beam's slot holds C blocks, one per k1, br_pitch(M)
// elements apart.  Between the launches a block holds for i = 0, 1, ... the pair's L
// elements as float4 {re, re, im, im}, then for R0 = 9 row 8 as complex values
// (launch 2 runs it with zeros beside it); launch 2 leaves the rows there as complex
// values: bin k1 + C (r0 + R0 q) is element q of row (k1, r0), at k1 br_pitch(M) +
// r0 L + q.  A slot's length (br_slot) does not depend on the plan: a batch's scratch
// is allocated once, and local sizes may change later.  (A whole row behind row 8,
// so that it runs as a pair like the others: 574 us for 577 on 1024 beams of 1000 ..
// 100000 samples, but slots of these plans a tenth longer than of others.)
//
// Where the last two passes multiply to 18 or less (972, 1458 and 864 points)
// launch 2 runs them in registers, one exchange fewer (rows 0.213 -> 0.20 ms on
// 1024 beams of 1000 .. 100000 samples).
//
// Why: one CTA per 16384-point row fills an SM's registers and shared memory, so
// loads, exchanges and stores take turns (39 % of the issue slots at 160
// instructions a point, clusters of up to 9 CTAs).  Items of 3000 .. 6000 points
// leave four CTAs per SM in different phases at half the instructions.  Bound:
// launch 1 by issue (42 % active; straight-line code of ~2000 instructions that
// each CTA runs once misses the instruction caches) and its loads' latency,
// launch 2 by the latency of its first loads and the L1's data path (57 %).
// Five CTAs per SM (96 registers, spills) 0.564 -> 0.588 ms on the same beams, not kept.
#pragma once

#include <type_traits>

#include "fft_core.cuh"
#include "fft_pair.cuh"

namespace spx {

// The local sizes taken: those of 16385 .. 147456-point 2^a 3^b transforms with a
// few per cent of the points each (the others keep the cluster kernel).
// R0: first radix; T: threads per row pair (64 or 128, a CTA has 128).
template <int M>
struct BrSize {
  static constexpr int R0 = CtPlan<M>::radix(0), L = M / R0, NP = (R0 + 1) / 2;
  static constexpr int T = (M == 16384 || M == 13824 || M == 12288) ? 64 : 128;
  // float4 entries of the passes' twiddles for one row pair
  static constexpr int rows(int p) { return CtPlan<M>::radix(p) == 4 ? 1 : CtPlan<M>::radix(p) - 1; }
  static constexpr int off(int p) { return p <= 1 ? 0 : off(p - 1) + rows(p - 1) * (CtPlan<M>::ns(p - 1) / R0); }
  static constexpr int entries = off(CtPlan<M>::npass);
};
constexpr bool br_size(uint32_t M) {
  return M == 16384 || M == 15552 || M == 13824 || M == 13122 || M == 12288 || M == 11664 || M == 6561;
}
// f(std::integral_constant<int, M>) for one of the sizes.
template <typename F>
__host__ __device__ __forceinline__ void br_switch(uint32_t M, F&& f) {
  switch (M) {
    case 16384: f(std::integral_constant<int, 16384>()); break;
    case 15552: f(std::integral_constant<int, 15552>()); break;
    case 13824: f(std::integral_constant<int, 13824>()); break;
    case 13122: f(std::integral_constant<int, 13122>()); break;
    case 12288: f(std::integral_constant<int, 12288>()); break;
    case 11664: f(std::integral_constant<int, 11664>()); break;
    default: f(std::integral_constant<int, 6561>()); break;
  }
}
constexpr uint32_t kBrThreads = 128;
// Elements from one k1's rows to the next one's: M up to 32-byte sectors.
__host__ __device__ constexpr uint32_t br_pitch(uint32_t M) { return (M + 3) & ~3u; }
// Elements of a beam's slot at whatever plan (of the local sizes only 6561 and its
// double are no multiples of 4).
constexpr uint32_t br_slot(uint32_t nfft) { return nfft + (nfft % 6561 == 0 ? 3 * (nfft / 6561) : 0u); }
constexpr uint32_t kBrMaxC = 9;
constexpr bool br_slots_fit() {
  for (uint32_t M = 6561; M <= 16384; ++M)
    for (uint32_t C = 2; br_size(M) && C <= kBrMaxC; ++C)
      if (C * br_pitch(M) > br_slot(C * M)) return false;
  return true;
}
static_assert(br_slots_fit(), "a slot holds its beam at every plan");

// ---- windows, two samples at a time ---------------------------------------------------
// window_at's operations (fft_core.cuh) on samples a and b, the polynomials in
// packed arithmetic: the same bits.  35 -> 18 instructions a sample (Hann).
// sin and cos of psi = (pi/2) s / D, s whole; (hi, lo) = (pi/2) / D.
SPX_DEV void sincos_small2(float2 s, float hi, float lo, float2* sn, float2* cs) {
  const float2 psi = pfma(s, pk(hi), pmul(s, pk(lo)));
  const float2 y = pmul(psi, psi);
  float2 c = pfma(y, pk(-1.0f / 3628800.0f), pk(1.0f / 40320.0f));
  c = pfma(c, y, pk(-1.0f / 720.0f));
  c = pfma(c, y, pk(1.0f / 24.0f));
  c = pfma(c, y, pk(-0.5f));
  *cs = pfma(c, y, pk(1.0f));
  float2 p = pfma(y, pk(1.0f / 362880.0f), pk(-1.0f / 5040.0f));
  p = pfma(p, y, pk(1.0f / 120.0f));
  p = pfma(p, y, pk(-1.0f / 6.0f));
  *sn = pfma(pmul(psi, y), p, psi);
}
// sin^2(pi n / D), n <= D: the angle 4 n / (2 D) quarter turns folds at D / 2 and
// back; only the square of the sine leaves, so no signs.
SPX_DEV float2 hann2(const WindowGen& g, uint32_t a, uint32_t b) {
  const uint32_t E = 2 * g.D;
  auto fold = [&](uint32_t n, bool* cosine) {
    const uint32_t t = 4 * n;
    const bool q = t >= E;
    const uint32_t r = q ? t - E : t;
    const bool swap = r > g.D;
    *cosine = swap != q;
    return __uint2float_rn(swap ? E - r : r);
  };
  bool ca, cb;
  const float sa = fold(a, &ca), sb = fold(b, &cb);
  float2 sn, cs;
  sincos_small2(make_float2(sa, sb), __fmul_rn(g.hi, 0.5f), __fmul_rn(g.lo, 0.5f), &sn, &cs);
  const float2 v = make_float2(ca ? cs.x : sn.x, cb ? cs.y : sn.y);
  return pmul(v, v);
}
SPX_DEV float2 cos2(const WindowGen& g, uint32_t k, uint32_t a, uint32_t b) {
  auto fold = [&](uint32_t n, bool* sine, bool* neg) {
    const uint32_t m4 = 4u * mul_mod(k, n, g.D);
    const uint32_t q = (uint32_t)(m4 >= g.D) + (uint32_t)(m4 >= 2u * g.D) + (uint32_t)(m4 >= 3u * g.D);
    const uint32_t r = m4 - q * g.D;
    const bool swap = 2u * r > g.D;
    *sine = swap != ((q & 1u) != 0);
    *neg = q == 1u || q == 2u;
    return __uint2float_rn(swap ? g.D - r : r);
  };
  bool ia, ib, na, nb;
  const float sa = fold(a, &ia, &na), sb = fold(b, &ib, &nb);
  float2 sn, cs;
  sincos_small2(make_float2(sa, sb), g.hi, g.lo, &sn, &cs);
  const float va = ia ? sn.x : cs.x, vb = ib ? sn.y : cs.y;
  return make_float2(na ? -va : va, nb ? -vb : vb);
}
SPX_DEV float2 window2(const WindowGen& g, uint32_t a, uint32_t b) {
  switch (g.kind) {
    case SPX_WINDOW_HANN: return hann2(g, a, b);
    case SPX_WINDOW_HAMMING: return pfma(pk(-0.46f), cos2(g, 1, a, b), pk(0.54f));
    case SPX_WINDOW_BLACKMAN:
      return pfma(pk(0.08f), cos2(g, 2, a, b), pfma(pk(-0.5f), cos2(g, 1, a, b), pk(0.42f)));
    case SPX_WINDOW_BLACKMAN_HARRIS:
      return pfma(pk(-0.01168f), cos2(g, 3, a, b),
                  pfma(pk(0.14128f), cos2(g, 2, a, b), pfma(pk(-0.48829f), cos2(g, 1, a, b), pk(0.35875f))));
    default: return pk(1.0f);
  }
}

// Sample n of a beam (0 from n_point on) and the beam's window.
struct BatchSamples {
  const float2* __restrict__ x;
  uint32_t n_point;
  WindowGen wg;
  SPX_DEV float2 operator()(uint32_t n) const { return n < n_point ? ld_stream(x + n) : make_float2(0.f, 0.f); }
};

// ---- launch 1 ----------------------------------------------------------------------
// Column pairs per tile: columns p and p + HW of 2 HW.
constexpr int br_hw(int C, int R0) { return R0 == 9 ? (C <= 4 ? 32 : 16) : C == 2 ? 64 : C <= 4 ? 32 : 16; }
// bytes of the largest tile (C = 9, R0 = 16) and its window values
constexpr uint32_t kBrTile = kBrMaxC * 16 * 16 * 16, kBrColsSmem = kBrTile + kBrTile / 2;

// The tile's window values are made by a loop of their own, into shared memory,
// while the samples' loads are in flight (the evaluation appears once, not
// unrolled into every load).
template <int C, int R0>
SPX_DEV void br_cols(float4* s4, const BatchSamples& load, uint32_t M, uint32_t L, uint32_t j0, const float2* __restrict__ twc,
                     float2* __restrict__ slot) {
  constexpr int HW = br_hw(C, R0), T = (int)kBrThreads, NI = R0 * HW, U = (NI + T - 1) / T, NP = R0 / 2;
  static_assert(C * R0 * HW * 16 <= (int)kBrTile, "tile");
  float2* wt = reinterpret_cast<float2*>(s4 + kBrTile / 16);  // [C R0][HW]: windows of columns p, p + HW
  const uint32_t tid = threadIdx.x;
  C2 v[U][C];
  // stage 1: item (p, r)
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = tid + u * T, p = i % HW, r = i / HW, ja = j0 + p, jb = ja + HW;
    if (NI % T == 0 || i < (uint32_t)NI) {
#pragma unroll
      for (int n1 = 0; n1 < C; ++n1) {
        const uint32_t n = M * n1 + L * r;
        const float2 a = ja < L ? load(n + ja) : make_float2(0.f, 0.f);
        const float2 b = jb < L ? load(n + jb) : make_float2(0.f, 0.f);
        v[u][n1] = C2{make_float2(a.x, b.x), make_float2(a.y, b.y)};
      }
    }
  }
  const bool windowed = load.wg.kind != SPX_WINDOW_NONE;
  if (windowed) {
#pragma unroll 1
    for (uint32_t i = tid; i < (uint32_t)(C * NI); i += T) {  // row i / HW: samples L (i / HW) + j
      const uint32_t a = L * (i / HW) + j0 + i % HW, b = a + HW;
      wt[i] = a < load.n_point ? window2(load.wg, a, min(b, load.wg.D)) : make_float2(0.f, 0.f);
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = tid + u * T, p = i % HW, r = i / HW, ja = j0 + p, jb = ja + HW;
    if (NI % T == 0 || i < (uint32_t)NI) {
      if (windowed) {  // (samples beyond n_point are 0 and stay 0)
#pragma unroll
        for (int n1 = 0; n1 < C; ++n1) {
          const float2 w = wt[(n1 * R0 + r) * HW + p];
          v[u][n1] = C2{pmul(v[u][n1].x, w), pmul(v[u][n1].y, w)};
        }
      }
      PDft<C>::run(v[u]);
      const float2 ta = __ldg(twc + L * r + min(ja, L - 1)), tb = __ldg(twc + L * r + min(jb, L - 1));
      C2 w[C];
      w[1] = C2{make_float2(ta.x, tb.x), make_float2(ta.y, tb.y)};
#pragma unroll
      for (int k1 = 2; k1 < C; ++k1) w[k1] = (k1 % 2 == 0) ? c2mul(w[k1 / 2], w[k1 / 2]) : c2mul(w[k1 - 1], w[1]);
#pragma unroll
      for (int k1 = 0; k1 < C; ++k1) {
        const C2 z = k1 == 0 ? v[u][0] : c2mul(v[u][k1], w[k1]);
        s4[(k1 * R0 + r) * HW + p] = make_float4(z.x.x, z.x.y, z.y.x, z.y.y);
      }
    }
  }
  __syncthreads();
  // stage 2: item (p, k1)
#pragma unroll 1
  for (uint32_t i = tid; i < (uint32_t)(C * HW); i += T) {
    const uint32_t p = i % HW, k1 = i / HW, ja = j0 + p, jb = ja + HW;
    C2 b[R0];
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      const float4 a = s4[(k1 * R0 + r) * HW + p];
      b[r] = C2{make_float2(a.x, a.y), make_float2(a.z, a.w)};
    }
    PDft<R0>::run(b);
    float2* block = slot + (size_t)k1 * br_pitch(M);
    float4* o = reinterpret_cast<float4*>(block);
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const C2 e = b[2 * q], f = b[2 * q + 1];
      if (ja < L) __stcg(o + (size_t)q * L + ja, make_float4(e.x.x, f.x.x, e.y.x, f.y.x));
      if (jb < L) __stcg(o + (size_t)q * L + jb, make_float4(e.x.y, f.x.y, e.y.y, f.y.y));
    }
    if constexpr (R0 % 2 != 0) {
      float2* r = block + (size_t)(R0 - 1) * L;
      if (ja < L) __stcg(r + ja, first_of(b[R0 - 1]));
      if (jb < L) __stcg(r + jb, second_of(b[R0 - 1]));
    }
  }
}

// ---- launch 2 ----------------------------------------------------------------------
// Pass P of the plan on one row pair by threads t < T: from the slots in device
// memory (the first; `alone`: src is one row of complex values), else from shared
// memory; the last hands element q of both rows to out(q, z).
template <int M, int P, typename Sync, typename Out>
SPX_DEV void br_pass(float4* s, const float2* src, bool alone, const float4* __restrict__ tw, uint32_t t,
                     const Out& out) {
  using PL = CtPlan<M>;
  using S = BrSize<M>;
  constexpr int T = S::T, R = PL::radix(P), Nr = PL::ns(P) / S::R0, B = S::L / R, Q = (B + T - 1) / T;
  constexpr bool first = P == 1, last = P == PL::npass - 1;
  const float4* tp = tw + S::off(P);
  auto have = [&](int q) { return B % T == 0 || q + 1 < Q || t + q * T < (uint32_t)B; };
  auto load = [&](C2* v, uint32_t j) {
    float4 a[R];
    if (first && S::R0 % 2 != 0 && alone) {  // (into the register pairs themselves: a wider load's moves would wait for it)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float* z = reinterpret_cast<const float*>(src + j + r * B);
        a[r] = make_float4(ld_value(z), 0.f, ld_value(z + 1), 0.f);
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = first ? ld_once4(src + 2 * (j + r * B)) : s[ps(j + r * B)];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = C2{make_float2(a[r].x, a[r].y), make_float2(a[r].z, a[r].w)};
  };
  auto butterfly = [&](C2* v, uint32_t k) {
    if constexpr (R == 4) {
      const C2 w1 = ld_tw(tp + k), w2 = c2mul(w1, w1);
      v[1] = c2mul(v[1], w1);
      v[2] = c2mul(v[2], w2);
      v[3] = c2mul(v[3], c2mul(w2, w1));
    } else {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = c2mul(v[r], ld_tw(tp + (r - 1) * Nr + k));
    }
    PDft<R>::run(v);
  };
  if constexpr (P >= 2 && P + 2 == PL::npass && R * PL::radix(P + 1) <= 18) {
    // the last two passes (R, then R2) in registers: the butterflies j = Nr a + k,
    // a < R2, of this pass share their twiddles and hold the inputs of the last
    // pass's butterflies Nr r + k
    constexpr int R2 = PL::radix(P + 1), Q2 = (Nr + T - 1) / T, N2 = Nr * R;
    const float4* tl = tw + S::off(P + 1);
#pragma unroll
    for (int q = 0; q < Q2; ++q) {
      const uint32_t k = t + q * T;
      if (!(Nr % T == 0 || q + 1 < Q2 || k < (uint32_t)Nr)) continue;
      C2 v[R2][R];
#pragma unroll
      for (int a = 0; a < R2; ++a) {
        load(v[a], Nr * a + k);
        butterfly(v[a], k);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        C2 w[R2];
#pragma unroll
        for (int a = 0; a < R2; ++a) w[a] = v[a][r];
        const uint32_t e = Nr * r + k;
        if constexpr (R2 == 4) {
          const C2 w1 = ld_tw(tl + e), w2 = c2mul(w1, w1);
          w[1] = c2mul(w[1], w1);
          w[2] = c2mul(w[2], w2);
          w[3] = c2mul(w[3], c2mul(w2, w1));
        } else {
#pragma unroll
          for (int a = 1; a < R2; ++a) w[a] = c2mul(w[a], ld_tw(tl + (a - 1) * N2 + e));
        }
        PDft<R2>::run(w);
#pragma unroll
        for (int a = 0; a < R2; ++a) out(e + N2 * a, w[a]);
      }
    }
  } else if constexpr (last) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!have(q)) continue;
      const uint32_t j = t + q * T;
      C2 v[R];
      load(v, j);
      butterfly(v, j);  // Nr = B: k = j
#pragma unroll
      for (int r = 0; r < R; ++r) out(j + r * B, v[r]);
    }
  } else {
    C2 v[Q][R];
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (have(q)) load(v[q], t + q * T);
    if constexpr (!first) Sync::wait();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (!have(q)) continue;
      const uint32_t j = t + q * T, k = j % Nr;
      butterfly(v[q], k);
      const uint32_t base = (j - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r)
        s[ps(base + r * Nr)] = make_float4(v[q][r].x.x, v[q][r].x.y, v[q][r].y.x, v[q][r].y.y);
    }
    Sync::wait();
    br_pass<M, P + 1, Sync>(s, src, alone, tw, t, out);
  }
}

// Slots of one row pair in shared memory.
template <int M>
constexpr uint32_t br_slots = BrSize<M>::L + (BrSize<M>::L + 15) / 16 + 1;
constexpr uint32_t kBrRowsSmem = 2 * (1024 + 65) * 16;  // the largest: two pairs of 1024
static_assert(br_slots<13122> * 16 <= kBrRowsSmem && 2 * br_slots<13824> * 16 <= kBrRowsSmem, "shared memory");

// Item k1 << 8 | j of a beam: row pair j of k1 (T = 128), or pairs 2 j and 2 j + 1.
// Elements [qlo, qhi) of the rows are left in the slot.
template <int M>
SPX_DEV void br_rows(float4* s4, uint32_t part, float2* __restrict__ slot, const float4* __restrict__ tables,
                     uint32_t qlo, uint32_t qhi) {
  using S = BrSize<M>;
  constexpr uint32_t L = S::L, T = S::T;
  const uint32_t t = threadIdx.x % T, h = threadIdx.x / T;
  const uint32_t k1 = part >> 8, i = (part & 255) * (kBrThreads / T) + h;
  const bool alone = S::R0 % 2 != 0 && i == S::NP - 1;
  float2* rows = slot + (size_t)k1 * br_pitch(M) + 2 * i * L;  // rows 2i and 2i + 1 of k1
  auto out = [=](uint32_t q, C2 z) {
    if (q >= qlo && q < qhi) {
      __stcg(rows + q, first_of(z));
      if (!alone) __stcg(rows + L + q, second_of(z));
    }
  };
  using Sync = std::conditional_t<T == kBrThreads, CtaSync, GroupSync<(int)T>>;
  br_pass<M, 1, Sync>(s4 + h * br_slots<M>, rows, alone, tables + i * S::entries, t, out);
}

}  // namespace spx
