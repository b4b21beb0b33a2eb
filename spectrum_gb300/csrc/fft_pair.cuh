// fft_pair.cuh — local FFTs of power-of-two size (1024 .. 16384 points) whose
// threads transform two neighbouring butterflies at once with packed FP32
// arithmetic (add/mul/fma on two values per instruction, sm_100 and later).
//
// The compile-time plans of fft_core.cuh (CtPlan: same radix order, same
// twiddle values, same operations in the same order on every element), so the
// results are the bits of ct_local_fft; what changes is the data layout:
//   * a register pair holds the same component of elements 2p and 2p + 1 (C2:
//     both real parts, both imaginary parts), so every addition,
//     multiplication and rotation by -i of two butterflies j = 2m, 2m + 1 is
//     one instruction (or none), and a twiddle product is four;
//   * shared memory holds 16-byte slots {re 2p, re 2p+1, im 2p, im 2p+1},
//     moved by 128-bit accesses: half the shared-memory instructions and
//     addresses per point;
//   * twiddle tables hold the pair W^{r k}, W^{r (k+1)} (k even) in the same
//     form, one 128-bit load for two points.
// In every pass but the first the outputs of butterflies 2m, 2m + 1 (an even
// stride) are neighbouring elements again; the first pass (stride 1) pairs the
// outputs r, r + 1 of one butterfly when it stores.
//
// Why: the scalar passes issue ~85 instructions per point and reach 45-55 % of
// the issue slots, with the FP32 pipe 30 % busy (ncu): issue slots and latency
// bound them, not memory.  The packed forms run at the FP32 pipe's full rate
// in half the issue slots (measured: 64 pair operations per clock and SM for
// add, mul and fma, operand negation free).
//
// Contraction: spx_device.cuh's Dft leaves mul/add contraction to the
// compiler; the forms below spell out the fused operations it chose (checked
// bit for bit on the GPU by tests/test_gpu_pair_fft.py against the scalar
// kernels).
#pragma once

#include "fft_core.cuh"

namespace spx {

// ---- packed arithmetic -------------------------------------------------------
SPX_DEV float2 pk(float k) { return make_float2(k, k); }
SPX_DEV float2 pneg(float2 a) { return make_float2(-a.x, -a.y); }
SPX_DEV float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
SPX_DEV float2 psub(float2 a, float2 b) { return __fadd2_rn(a, pneg(b)); }
SPX_DEV float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
SPX_DEV float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Two complex values: real parts and imaginary parts of elements 2p, 2p + 1.
struct C2 {
  float2 x, y;
};
SPX_DEV float2 first_of(C2 z) { return make_float2(z.x.x, z.y.x); }
SPX_DEV float2 second_of(C2 z) { return make_float2(z.x.y, z.y.y); }
SPX_DEV C2 c2add(C2 a, C2 b) { return C2{padd(a.x, b.x), padd(a.y, b.y)}; }
SPX_DEV C2 c2sub(C2 a, C2 b) { return C2{psub(a.x, b.x), psub(a.y, b.y)}; }
// a * w, the operations of cmul on both values
SPX_DEV C2 c2mul(C2 a, C2 w) {
  return C2{pfma(a.x, w.x, pneg(pmul(a.y, w.y))), pfma(a.x, w.y, pmul(a.y, w.x))};
}
// a * (wx + i wy), constants
SPX_DEV C2 c2mulc(C2 a, float wx, float wy) {
  return C2{pfma(a.x, pk(wx), pmul(a.y, pk(-wy))), pfma(a.x, pk(wy), pmul(a.y, pk(wx)))};
}

SPX_DEV void pdft4_tail(C2 s02, C2 d02, C2 s13, C2 d13, C2& a0, C2& a1, C2& a2, C2& a3) {
  a0 = c2add(s02, s13);
  a2 = c2sub(s02, s13);
  a1 = C2{padd(d02.x, d13.y), psub(d02.y, d13.x)};  // d02 - i*d13
  a3 = C2{psub(d02.x, d13.y), padd(d02.y, d13.x)};  // d02 + i*d13
}
SPX_DEV void pdft4(C2& a0, C2& a1, C2& a2, C2& a3) {
  pdft4_tail(c2add(a0, a2), c2sub(a0, a2), c2add(a1, a3), c2sub(a1, a3), a0, a1, a2, a3);
}

template <int R>
struct PDft;

template <>
struct PDft<2> {
  static SPX_DEV void run(C2* v) {
    const C2 t = v[0];
    v[0] = c2add(t, v[1]);
    v[1] = c2sub(t, v[1]);
  }
};
template <>
struct PDft<4> {
  static SPX_DEV void run(C2* v) { pdft4(v[0], v[1], v[2], v[3]); }
};
SPX_DEV void pdft3(C2& a0, C2& a1, C2& a2) {
  const C2 t = c2add(a1, a2), u = c2sub(a1, a2);
  const C2 m{pfma(pk(-0.5f), t.x, a0.x), pfma(pk(-0.5f), t.y, a0.y)};
  const float2 k = pk(kS3), nk = pk(-kS3);
  a0 = c2add(a0, t);
  a1 = C2{pfma(u.y, k, m.x), pfma(u.x, nk, m.y)};  // m - i k u
  a2 = C2{pfma(u.y, nk, m.x), pfma(u.x, k, m.y)};  // m + i k u
}
template <>
struct PDft<3> {
  static SPX_DEV void run(C2* v) { pdft3(v[0], v[1], v[2]); }
};
template <>
struct PDft<6> {
  static SPX_DEV void run(C2* v) {
    C2 e0 = v[0], e1 = v[2], e2 = v[4], o0 = v[1], o1 = v[3], o2 = v[5];
    pdft3(e0, e1, e2);
    pdft3(o0, o1, o2);
    o1 = c2mulc(o1, 0.5f, -kS3);
    o2 = c2mulc(o2, -0.5f, -kS3);
    v[0] = c2add(e0, o0);
    v[3] = c2sub(e0, o0);
    v[1] = c2add(e1, o1);
    v[4] = c2sub(e1, o1);
    v[2] = c2add(e2, o2);
    v[5] = c2sub(e2, o2);
  }
};
template <>
struct PDft<9> {
  static SPX_DEV void run(C2* v) {
    // columns n2: v[n2], v[n2 + 3], v[n2 + 6] -> b[n2][k1] in place
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) pdft3(v[n2], v[3 + n2], v[6 + n2]);
    auto b = [&](int n2, int k1) -> C2& { return v[3 * k1 + n2]; };
    b(1, 1) = c2mulc(b(1, 1), kC9a, -kS9a);
    b(1, 2) = c2mulc(b(1, 2), kC9b, -kS9b);
    b(2, 1) = c2mulc(b(2, 1), kC9b, -kS9b);
    b(2, 2) = c2mulc(b(2, 2), -kC9c, -kS9c);
    C2 o[9];
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      C2 a0 = b(0, k1), a1 = b(1, k1), a2 = b(2, k1);
      pdft3(a0, a1, a2);
      o[k1] = a0;
      o[k1 + 3] = a1;
      o[k1 + 6] = a2;
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = o[i];
  }
};
template <>
struct PDft<12> {
  static SPX_DEV void run(C2* v) {
    // columns n2: v[n2], v[n2 + 4], v[n2 + 8] -> b[n2][k1] in place
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) pdft3(v[n2], v[4 + n2], v[8 + n2]);
    auto b = [&](int n2, int k1) -> C2& { return v[4 * k1 + n2]; };
    b(1, 1) = c2mulc(b(1, 1), kS3, -0.5f);
    b(1, 2) = c2mulc(b(1, 2), 0.5f, -kS3);
    b(2, 1) = c2mulc(b(2, 1), 0.5f, -kS3);
    b(2, 2) = c2mulc(b(2, 2), -0.5f, -kS3);
    b(3, 1) = C2{b(3, 1).y, pneg(b(3, 1).x)};
    b(3, 2) = C2{pneg(b(3, 2).x), pneg(b(3, 2).y)};
    C2 o[12];
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      C2 a0 = b(0, k1), a1 = b(1, k1), a2 = b(2, k1), a3 = b(3, k1);
      pdft4(a0, a1, a2, a3);
      o[k1] = a0;
      o[k1 + 3] = a1;
      o[k1 + 6] = a2;
      o[k1 + 9] = a3;
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) v[i] = o[i];
  }
};
template <>
struct PDft<8> {
  static SPX_DEV void run(C2* v) {
    C2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    C2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    pdft4(e0, e1, e2, e3);
    pdft4(o0, o1, o2, o3);
    // o1 (1 - i)/sqrt2 = k t1, o2 (-i), o3 (-1 - i)/sqrt2 = k (t3.x, -t3.y)
    const C2 t1{padd(o1.x, o1.y), psub(o1.y, o1.x)};
    const C2 t3{psub(o3.y, o3.x), padd(o3.x, o3.y)};
    const float2 k = pk(kS2), nk = pk(-kS2);
    v[0] = c2add(e0, o0);
    v[4] = c2sub(e0, o0);
    v[1] = C2{pfma(t1.x, k, e1.x), pfma(t1.y, k, e1.y)};
    v[5] = C2{pfma(t1.x, nk, e1.x), pfma(t1.y, nk, e1.y)};
    v[2] = C2{padd(e2.x, o2.y), psub(e2.y, o2.x)};
    v[6] = C2{psub(e2.x, o2.y), padd(e2.y, o2.x)};
    v[3] = C2{pfma(t3.x, k, e3.x), pfma(t3.y, nk, e3.y)};
    v[7] = C2{pfma(t3.x, nk, e3.x), pfma(t3.y, k, e3.y)};
  }
};
template <>
struct PDft<16> {
  static SPX_DEV void run(C2* v) {
    // columns n2: v[n2], v[n2 + 4], v[n2 + 8], v[n2 + 12] -> b[n2][k1] in place
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) pdft4(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    const float2 k = pk(kS2), nk = pk(-kS2);
    auto b = [&](int n2, int k1) -> C2& { return v[4 * k1 + n2]; };
    b(1, 1) = c2mulc(b(1, 1), kC16, -kS16);
    b(1, 3) = c2mulc(b(1, 3), kS16, -kC16);
    b(3, 1) = c2mulc(b(3, 1), kS16, -kC16);
    b(3, 3) = c2mulc(b(3, 3), -kC16, kS16);
    // the rotations by odd multiples of pi/4 leave their factor k to the sums
    C2 o[4][4];
    {  // k1 = 0
      C2 a0 = b(0, 0), a1 = b(1, 0), a2 = b(2, 0), a3 = b(3, 0);
      pdft4(a0, a1, a2, a3);
      o[0][0] = a0; o[0][1] = a1; o[0][2] = a2; o[0][3] = a3;
    }
    {  // k1 = 1: a2 = k (t.x, t.y)
      const C2 z = b(2, 1), a0 = b(0, 1);
      const C2 t{padd(z.x, z.y), psub(z.y, z.x)};
      pdft4_tail(C2{pfma(t.x, k, a0.x), pfma(t.y, k, a0.y)}, C2{pfma(t.x, nk, a0.x), pfma(t.y, nk, a0.y)},
                 c2add(b(1, 1), b(3, 1)), c2sub(b(1, 1), b(3, 1)), o[1][0], o[1][1], o[1][2], o[1][3]);
    }
    {  // k1 = 2: a1 = k (P.x, P.y), a2 = -i z, a3 = k (Q.x, -Q.y)
      const C2 z1 = b(1, 2), z = b(2, 2), z3 = b(3, 2), a0 = b(0, 2);
      const C2 P{padd(z1.x, z1.y), psub(z1.y, z1.x)}, Q{psub(z3.y, z3.x), padd(z3.x, z3.y)};
      const float2 qx = pmul(Q.x, k), qy = pmul(Q.y, k);
      pdft4_tail(C2{padd(a0.x, z.y), psub(a0.y, z.x)}, C2{psub(a0.x, z.y), padd(a0.y, z.x)},
                 C2{pfma(P.x, k, qx), pfma(P.y, k, pneg(qy))}, C2{pfma(P.x, k, pneg(qx)), pfma(P.y, k, qy)},
                 o[2][0], o[2][1], o[2][2], o[2][3]);
    }
    {  // k1 = 3: a2 = k (t.x, -t.y)
      const C2 z = b(2, 3), a0 = b(0, 3);
      const C2 t{psub(z.y, z.x), padd(z.x, z.y)};
      pdft4_tail(C2{pfma(t.x, k, a0.x), pfma(t.y, nk, a0.y)}, C2{pfma(t.x, nk, a0.x), pfma(t.y, k, a0.y)},
                 c2add(b(1, 3), b(3, 3)), c2sub(b(1, 3), b(3, 3)), o[3][0], o[3][1], o[3][2], o[3][3]);
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = o[k1][k2];
  }
};

// ---- shared-memory layout ------------------------------------------------------
// Slot p (elements 2p, 2p + 1) at ps(p) = p + p/16: a quarter-warp's eight
// 128-bit accesses hit eight different 16-byte banks for unit strides (every
// pass's loads and the stores of strides >= 16) and for the stride-16 stores
// of a first radix-16 pass.
SPX_DEV uint32_t ps(uint32_t p) { return p + (p >> 4); }
// 16-byte slots of an M-point local FFT (the bytes of sw_len(M) elements).
constexpr uint32_t ps_len(uint32_t M) { return M / 2 + M / 32; }
// Element i of the natural-order result in shared memory.
SPX_DEV float2 pair_elem(const float4* s, uint32_t i) {
  const float* f = reinterpret_cast<const float*>(s + ps(i >> 1)) + (i & 1u);
  return make_float2(f[0], f[2]);
}

// ---- plans -----------------------------------------------------------------------
// Entries (float4) of a pass's pair table: per twiddle row, Ns / 2 pairs; a
// split radix-4 pass holds 32 pairs W^l, W^{l+1} (l < 64), then W^{64 j}
// twice over (both values the same).
constexpr uint32_t pair_tw_entries(uint32_t R, uint32_t Ns) {
  return Ns < 2 ? 0u : tw_split(R, Ns) ? 32u + Ns / 64u : tw_rows(R) * (Ns / 2);
}
constexpr bool pair_size(uint32_t M) { return M >= 1024 && M <= 16384 && (M & (M - 1)) == 0; }

template <int M>
struct PairPlan : CtPlan<M> {
  static_assert(pair_size((uint32_t)M), "power of two, 1024 .. 16384");
  using P0 = CtPlan<M>;
  static constexpr int T = M / 32;  // threads: two radix-16 butterflies each
  static constexpr int ptwoff(int p) {
    return p == 0 ? 0 : ptwoff(p - 1) + (int)pair_tw_entries((uint32_t)P0::radix(p - 1), (uint32_t)P0::ns(p - 1));
  }
};

// ---- loads -------------------------------------------------------------------------
SPX_DEV float4 ld_stream4(const float2* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Two complex values that are read once (not kept in L1, which holds the
// twiddles): memory this launch may write later, so not the read-only path.
SPX_DEV float4 ld_once4(const void* p) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
SPX_DEV float ld_value(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// Two table values (volatile: issued where it stands).
SPX_DEV float2 ld_table2(const float* p) {
  float2 v;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// Samples n, n + 1 (n even) of a beam: window applied (load_sample's rounded
// multiplies), zero beyond n_point.  16-byte loads when the beam starts on a
// 16-byte boundary and n_point is even (no pair then straddles the end), else
// two 8-byte loads that keep the line in L1 for the second.  Window values come
// in pairs on both paths (n is even; the table has a zero behind its last value),
// all of them and the samples in flight before the first product: read one by one
// between the products, 64 x 2^19 points 8 bytes off a boundary took 297 us instead
// of 226, 8192 x 4096 points 140 instead of 95.  The products stand once behind both
// paths: the kernels are long and run once per CTA, and instruction fetch counts
// (two copies: 256 x 131072 points 226 us for 214, 64 x 2^19 241 for 225).
struct SamplePairs {
  const float2* __restrict__ x;
  uint32_t n_point;
  const float* __restrict__ win;
  bool vec;
  SPX_DEV SamplePairs(const float2* x_, uint32_t n, const float* w)
      : x(x_), n_point(n), win(w), vec(((reinterpret_cast<uintptr_t>(x_) & 15u) | (n & 1u)) == 0) {}
  template <int R>
  SPX_DEV void load(C2 (&v)[R], uint32_t n0, uint32_t step) const {
    float4 a[R];
    if (win) {
      float2 w[R];
      if (vec) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t n = n0 + r * step;
          a[r] = make_float4(0.f, 0.f, 0.f, 0.f);
          w[r] = make_float2(0.f, 0.f);
          if (n < n_point) {
            a[r] = ld_stream4(x + n);
            w[r] = ld_table2(win + n);
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t n = n0 + r * step;
          float2 b = make_float2(0.f, 0.f), c = b;
          w[r] = b;
          if (n < n_point) {
            b = ld_table2(reinterpret_cast<const float*>(x + n));
            w[r] = ld_table2(win + n);
          }
          if (n + 1 < n_point) c = ld_table2(reinterpret_cast<const float*>(x + n + 1));
          a[r] = make_float4(b.x, b.y, c.x, c.y);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (n0 + r * step < n_point)
          a[r] = make_float4(__fmul_rn(a[r].x, w[r].x), __fmul_rn(a[r].y, w[r].x), __fmul_rn(a[r].z, w[r].y),
                             __fmul_rn(a[r].w, w[r].y));
    } else if (vec) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t n = n0 + r * step;
        a[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < n_point) a[r] = ld_stream4(x + n);
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t n = n0 + r * step;
        const float2 b = n < n_point ? __ldg(x + n) : make_float2(0.f, 0.f);
        const float2 c = n + 1 < n_point ? __ldg(x + n + 1) : make_float2(0.f, 0.f);
        a[r] = make_float4(b.x, b.y, c.x, c.y);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = C2{make_float2(a[r].x, a[r].z), make_float2(a[r].y, a[r].w)};
  }
};

// Samples of a chirp-z transform: SamplePairs times the chirp w[n], n < n_point
// (chirp_pre_kernel's product), zero beyond.  w is readable up to an even count.
struct ChirpPairs {
  SamplePairs x;
  const float2* __restrict__ w;
  template <int R>
  SPX_DEV void load(C2 (&v)[R], uint32_t n0, uint32_t step) const {
    x.load(v, n0, step);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t n = n0 + r * step;
      if (n < x.n_point) {
        const float4 c = __ldg(reinterpret_cast<const float4*>(w + n));
        const C2 z = c2mul(v[r], C2{make_float2(c.x, c.z), make_float2(c.y, c.w)});
        const bool both = n + 1 < x.n_point;
        v[r] = C2{make_float2(z.x.x, both ? z.x.y : 0.f), make_float2(z.y.x, both ? z.y.y : 0.f)};
      }
    }
  }
};

// Elements n, n + 1 of a row written earlier by other CTAs (exchange slots):
// L2-coherent 16-byte loads (rows start on 16-byte boundaries).  LAST: no one reads
// the row again, and it leaves the L2 first.
template <bool LAST = false>
struct ExchangePairs {
  const float2* row;
  template <int R>
  SPX_DEV void load(C2 (&v)[R], uint32_t n0, uint32_t step) const {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4* p = reinterpret_cast<const float4*>(row + n0 + r * step);
      const float4 a = LAST ? __ldcs(p) : __ldcg(p);
      v[r] = C2{make_float2(a.x, a.z), make_float2(a.y, a.w)};
    }
  }
};

// ---- passes ------------------------------------------------------------------------
// Outputs of butterflies 2m, 2m + 1 of a first pass: slots m R + r/2 and
// m R + R/2 + r/2 (r even); R = 16: ps(16 m + c) = 17 m + c (c < 16); R = 8:
// 8 m + m/2 + c (c < 8).
template <int R>
SPX_DEV void pair_first_store(float4* s, uint32_t m, const C2* v) {
  static_assert(R == 16 || R == 8, "first radix");
  float4* d = s + (R == 16 ? 17 * m : 8 * m + (m >> 1));
#pragma unroll
  for (int r = 0; r < R; r += 2) {
    d[r / 2] = make_float4(v[r].x.x, v[r + 1].x.x, v[r].y.x, v[r + 1].y.x);
    d[R / 2 + r / 2] = make_float4(v[r].x.y, v[r + 1].x.y, v[r].y.y, v[r + 1].y.y);
  }
}

template <int M, int T, typename Sync = CtaSync, typename Load>
SPX_DEV void pair_first(float4* s, const Load& load, uint32_t tid) {
  constexpr int R = CtPlan<M>::radix(0), B = M / R, Q = B / 2 / T;
  static_assert(R % 2 == 0 && Q * 2 * T == B, "whole pairs");
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint32_t m = tid + q * T;
    C2 v[R];
    load.load(v, 2 * m, B);
    PDft<R>::run(v);
    pair_first_store<R>(s, m, v);
  }
  Sync::wait();
}

SPX_DEV C2 ld_tw(const float4* __restrict__ t) {
  const float4 w = __ldg(t);
  return C2{make_float2(w.x, w.y), make_float2(w.z, w.w)};
}

// Loads and twiddles of the butterflies 2m, 2m + 1 of pass P, then their DFT.
template <int M, int P>
SPX_DEV void pair_load(const float4* s, C2* v, uint32_t m) {
  constexpr int R = CtPlan<M>::radix(P), H = M / R / 2;  // slots between inputs
  static_assert(H % 16 == 0, "constant slot offsets");
  const float4* p = s + ps(m);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float4 a = p[r * (H + H / 16)];
    v[r] = C2{make_float2(a.x, a.y), make_float2(a.z, a.w)};
  }
}
template <int M, int P>
SPX_DEV void pair_butterfly(C2* v, const float4* __restrict__ tw, uint32_t m) {
  constexpr int R = CtPlan<M>::radix(P), Ns = CtPlan<M>::ns(P);
  const uint32_t kk = m & (Ns / 2 - 1);  // k / 2
  const float4* t = tw + PairPlan<M>::ptwoff(P);
  if constexpr (R == 4) {
    C2 w1;
    if constexpr (tw_split(4, Ns))
      w1 = c2mul(ld_tw(t + 32 + (kk >> 5)), ld_tw(t + (kk & 31u)));
    else
      w1 = ld_tw(t + kk);
    const C2 w2 = c2mul(w1, w1);
    v[1] = c2mul(v[1], w1);
    v[2] = c2mul(v[2], w2);
    v[3] = c2mul(v[3], c2mul(w2, w1));
  } else {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = c2mul(v[r], ld_tw(t + (r - 1) * (Ns / 2) + kk));
  }
  PDft<R>::run(v);
}

// First pass from the slots themselves (the natural-order result of an earlier
// transform, behind a barrier): every load before the first store.
template <int M, int T>
SPX_DEV void pair_first_slots(float4* s, uint32_t tid) {
  constexpr int R = CtPlan<M>::radix(0), Q = M / R / 2 / T;
  C2 v[Q][R];
#pragma unroll
  for (int q = 0; q < Q; ++q) pair_load<M, 0>(s, v[q], tid + q * T);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    PDft<R>::run(v[q]);
    pair_first_store<R>(s, tid + q * T, v[q]);
  }
  __syncthreads();
}

// Pass P (not the first, not the last) in shared memory.
template <int M, int P, int T, typename Sync = CtaSync>
SPX_DEV void pair_pass(float4* s, const float4* __restrict__ tw, uint32_t tid) {
  constexpr int R = CtPlan<M>::radix(P), Ns = CtPlan<M>::ns(P), Q = M / R / 2 / T, H = Ns / 2;
  static_assert(Q == 1, "one pair of butterflies per thread");
  C2 v[R];
  pair_load<M, P>(s, v, tid);
  Sync::wait();
  pair_butterfly<M, P>(v, tw, tid);
  // slot of output r: ((j - k) R + k) / 2 + r H with j = 2m; H divides 16 or is a multiple of it
  const uint32_t kk = tid & (H - 1);
  float4* d = s + ps((tid - kk) * R + kk);
#pragma unroll
  for (int r = 0; r < R; ++r)
    d[r * H + ((r * H) >> 4)] = make_float4(v[r].x.x, v[r].x.y, v[r].y.x, v[r].y.y);
  Sync::wait();
}
template <int M, int P, int T, typename Sync = CtaSync>
SPX_DEV void pair_passes_until_last(float4* s, const float4* __restrict__ tw, uint32_t tid) {
  if constexpr (P + 1 < CtPlan<M>::npass) {
    pair_pass<M, P, T, Sync>(s, tw, tid);
    pair_passes_until_last<M, P + 1, T, Sync>(s, tw, tid);
  }
}

// Last pass: out(i, z) takes elements i, i + 1 (i even) of the natural-order
// result; consecutive threads get consecutive pairs.  Ends without a barrier.
template <int M, int T, typename Out>
SPX_DEV void pair_last(const float4* s, const float4* __restrict__ tw, uint32_t tid, const Out& out) {
  constexpr int P = CtPlan<M>::npass - 1;
  constexpr int R = CtPlan<M>::radix(P), B = M / R, Q = B / 2 / T;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint32_t m = tid + q * T;
    C2 v[R];
    pair_load<M, P>(s, v, m);
    pair_butterfly<M, P>(v, tw, m);
#pragma unroll
    for (int r = 0; r < R; ++r) out(2 * m + r * B, v[r]);
  }
}

// The whole local FFT (M / 32 threads): first pass from `load`, the result
// handed to out(i, z) (pair_last); ends without a barrier.
template <int M, typename Load, typename Out>
SPX_DEV void pair_local_fft_out(float4* s, const Load& load, const float4* __restrict__ tw, uint32_t tid,
                                const Out& out) {
  constexpr int T = PairPlan<M>::T;
  pair_first<M, T>(s, load, tid);
  pair_passes_until_last<M, 1, T>(s, tw, tid);
  pair_last<M, T>(s, tw, tid, out);
}

// ---- 8192 points -------------------------------------------------------------------
// Radices 16, 16, 16, 2.  Here a pair is an element and its neighbour at the
// distance of the NEXT stride: the butterflies j, j + Ns of a pass share their
// twiddles (one 8-byte load for both) and leave their outputs r as elements e,
// e + 16 Ns, the next pass's pairs, so the first pass stores its registers as
// they are, and the third leaves elements e, e + 4096: the last pass's
// butterflies, finished in registers.  Two exchanges instead of three.
// (16384 points end in a radix-4 pass over two pairs, 4096 in a radix-16 pass
// over eight: their last pass would be scalar, which costs more than the pairs
// of neighbours do.)
//   pass 0: butterflies 2m, 2m + 1      -> elements 32 m + r, + 16: slot 16 m + r
//   pass 1: j = 32 a + k and j + 16     -> elements 512 a + 16 r + k, + 256: slot 256 a + 16 r + k
//   pass 2: j = k and j + 256           -> elements k + 256 r, + 4096: slot 256 r + k
// out(e, z0, z1) takes elements e and e + 4096.
SPX_DEV C2 tw_both(const float2* __restrict__ t) {  // one twiddle for both values
  const float2 w = __ldg(t);
  return C2{pk(w.x), pk(w.y)};
}
template <typename Load, typename Out>
SPX_DEV void pair8k_fft_out(float4* s, const Load& load, const float2* __restrict__ tw, uint32_t tid, const Out& out) {
  using P = CtPlan<8192>;
  static_assert(P::npass == 4 && P::radix(0) == 16 && P::radix(1) == 16 && P::radix(2) == 16 && P::radix(3) == 2, "plan");
  constexpr uint32_t step = 256 + 16;  // slots between a pass's inputs
  C2 v[16];
  load.load(v, 2 * tid, 512);
  PDft<16>::run(v);
#pragma unroll
  for (int r = 0; r < 16; ++r) s[17 * tid + r] = make_float4(v[r].x.x, v[r].x.y, v[r].y.x, v[r].y.y);
  __syncthreads();
  const float4* p = s + ps(tid);
#pragma unroll
  for (int q = 1; q <= 2; ++q) {
    const uint32_t Ns = q == 1 ? 16 : 256, k = tid & (Ns - 1);
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const float4 a = p[r * step];
      v[r] = C2{make_float2(a.x, a.y), make_float2(a.z, a.w)};
    }
    if (q == 1) __syncthreads();
    const float2* t = tw + P::twoff(q) + k;
#pragma unroll
    for (int r = 1; r < 16; ++r) v[r] = c2mul(v[r], tw_both(t + (r - 1) * Ns));
    PDft<16>::run(v);
    if (q == 1) {
      float4* d = s + ps(256 * (tid >> 4)) + k;
#pragma unroll
      for (int r = 0; r < 16; ++r) d[17 * r] = make_float4(v[r].x.x, v[r].x.y, v[r].y.x, v[r].y.y);
      __syncthreads();
    }
  }
  if constexpr (Out::kMoves) __syncthreads();  // (every input read before the first output)
  // (the last twiddles all in flight before the outputs, whose square roots
  // would keep the compiler from issuing them early)
  float2 w[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) w[r] = ld_table2(reinterpret_cast<const float*>(tw + P::twoff(3) + tid + 256 * r));
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    const float2 a = first_of(v[r]), b = cmul(second_of(v[r]), w[r]);
    out(tid + 256 * r, cadd(a, b), csub(a, b));
  }
}

// Result in natural order (element i is the i-th float2; not the slots' layout),
// elements beyond `last` left out.
struct Natural8kOut {
  static constexpr bool kMoves = true;  // other slots than this thread read
  float2* s;
  uint32_t last;
  SPX_DEV void operator()(uint32_t e, float2 a, float2 b) const {
    s[e] = a;
    if (e + 4096 <= last) s[e + 4096] = b;
  }
};

// Result back into the slots it was read from (element i at pair_elem(s, i));
// SlotOutUpTo leaves elements beyond `last` out.
struct SlotOut {
  float4* s;
  SPX_DEV void operator()(uint32_t i, C2 z) const { s[ps(i >> 1)] = make_float4(z.x.x, z.x.y, z.y.x, z.y.y); }
};
struct SlotOutUpTo {
  float4* s;
  uint32_t last;
  SPX_DEV void operator()(uint32_t i, C2 z) const {
    if (i <= last) SlotOut{s}(i, z);
  }
};

// ---- outputs -------------------------------------------------------------------------

// Output of bins i, i + 1 of one beam's natural-order spectrum (the layouts
// of store_bin); `out` is 16-byte aligned (8 bytes for magnitudes).
template <int M, int MODE>
struct BinOutPairs;
constexpr int kPairComplex = 0, kPairMag = 1, kPairMagPhase = 2, kPairReversed = 3, kPairOther = 4;

template <int M>
struct BinOutPairs<M, kPairComplex> {
  float4* row;
  SPX_DEV BinOutPairs(void* out, uint32_t, float, const FftGeom&, uint32_t beam)
      : row(reinterpret_cast<float4*>(out) + (size_t)beam * (M / 2)) {}
  SPX_DEV void operator()(uint32_t i, C2 z) const { row[i >> 1] = make_float4(z.x.x, z.y.x, z.x.y, z.y.y); }
};
template <int M>
struct BinOutPairs<M, kPairMag> {  // |X| or |X|^2, times scale
  float2* row;
  bool squared;
  float scale;
  SPX_DEV BinOutPairs(void* out, uint32_t mode, float sc, const FftGeom&, uint32_t beam)
      : row(reinterpret_cast<float2*>(out) + (size_t)beam * (M / 2)), squared(mode == SPX_OUT_MAG2), scale(sc) {}
  SPX_DEV void operator()(uint32_t i, C2 z) const {
    float a = mag2_rn(first_of(z)), b = mag2_rn(second_of(z));
    if (!squared) {
      a = __fsqrt_rn(a);
      b = __fsqrt_rn(b);
    }
    row[i >> 1] = make_float2(__fmul_rn(a, scale), __fmul_rn(b, scale));
  }
};
template <int M>
struct BinOutPairs<M, kPairMagPhase> {
  float4* row;
  SPX_DEV BinOutPairs(void* out, uint32_t, float, const FftGeom&, uint32_t beam)
      : row(reinterpret_cast<float4*>(out) + (size_t)beam * (M / 2)) {}
  SPX_DEV void operator()(uint32_t i, C2 z) const {
    const float2 a = first_of(z), b = second_of(z);
    row[i >> 1] = make_float4(mag_rn(a), atan2f(a.y, a.x), mag_rn(b), atan2f(b.y, b.x));
  }
};
// Inverse transform: bin k goes to element (M - k) mod M, scaled.  A pair of
// elements (p, p + 1), p even, holds bins i + 2 and i + 1 (p = M - i - 2): the
// first comes from the next lane; the warp's ends are stored alone.
template <int M>
struct BinOutPairs<M, kPairReversed> {
  float2* row;
  float scale;
  SPX_DEV BinOutPairs(void* out, uint32_t, float sc, const FftGeom&, uint32_t beam)
      : row(reinterpret_cast<float2*>(out) + (size_t)beam * M), scale(sc) {}
  SPX_DEV void operator()(uint32_t i, C2 z) const {
    const uint32_t lane = threadIdx.x & 31u;
    const float2 a = make_float2(__fmul_rn(z.x.x, scale), __fmul_rn(z.y.x, scale));
    const float2 b = make_float2(__fmul_rn(z.x.y, scale), __fmul_rn(z.y.y, scale));
    const float nx = __shfl_down_sync(0xffffffffu, a.x, 1), ny = __shfl_down_sync(0xffffffffu, a.y, 1);
    if (lane == 0) row[i == 0 ? 0u : M - i] = a;
    if (lane == 31)
      row[M - i - 1] = b;
    else
      *reinterpret_cast<float4*>(row + (M - i - 2)) = make_float4(nx, ny, b.x, b.y);
  }
};
template <int M>
struct BinOutPairs<M, kPairOther> {  // any mode, any alignment
  void* out;
  uint32_t mode, beam;
  float scale;
  const FftGeom& g;
  SPX_DEV BinOutPairs(void* o, uint32_t m, float sc, const FftGeom& gg, uint32_t b)
      : out(o), mode(m), beam(b), scale(sc), g(gg) {}
  SPX_DEV void operator()(uint32_t i, C2 z) const {
    store_bin(out, mode, scale, g, beam, i, first_of(z));
    store_bin(out, mode, scale, g, beam, i + 1, second_of(z));
  }
};

// Output of elements e and e + 4096 of an 8192-point transform (8192-point
// specialisations of the modes above; every store of a warp is contiguous).
template <int MODE>
struct BinOut8k {
  static constexpr bool kMoves = false;
  void* out;
  uint32_t mode, beam;
  float scale;
  const FftGeom& g;
  SPX_DEV void one(uint32_t k, float2 z) const {
    const size_t at = (size_t)beam * 8192 + k;
    if constexpr (MODE == kPairComplex) {
      reinterpret_cast<float2*>(out)[at] = z;
    } else if constexpr (MODE == kPairMag) {
      const float m2 = mag2_rn(z);
      reinterpret_cast<float*>(out)[at] = __fmul_rn(mode == SPX_OUT_MAG2 ? m2 : __fsqrt_rn(m2), scale);
    } else if constexpr (MODE == kPairMagPhase) {
      reinterpret_cast<float2*>(out)[at] = make_float2(mag_rn(z), atan2f(z.y, z.x));
    } else if constexpr (MODE == kPairReversed) {
      reinterpret_cast<float2*>(out)[(size_t)beam * 8192 + ((8192 - k) & 8191)] =
          make_float2(__fmul_rn(z.x, scale), __fmul_rn(z.y, scale));
    } else {
      store_bin(out, mode, scale, g, beam, k, z);
    }
  }
  SPX_DEV void operator()(uint32_t e, float2 a, float2 b) const {
    one(e, a);
    one(e + 4096, b);
  }
};

// ---- cross stage -----------------------------------------------------------------------
// cross_stage_exchange for two neighbouring columns n2, n2 + 1 per thread
// (CR a power of two, M / CR even): the same operations on each column.
template <int CR, int M, int T>
SPX_DEV void pair_cross_stage(float2* __restrict__ slot, uint32_t c, const SamplePairs& load,
                              const float2* __restrict__ twc, uint32_t tid) {
  constexpr uint32_t S = M / CR;
  static_assert(S % 2 == 0 && (S / 2) % T == 0, "whole pairs of columns");
#pragma unroll 1
  for (uint32_t q = tid; q < S / 2; q += T) {
    const uint32_t n2 = c * S + 2 * q;
    C2 v[CR];
    load.load(v, n2, M);
    const float4 t = __ldg(reinterpret_cast<const float4*>(twc + n2));
    PDft<CR>::run(v);
    auto put = [&](int k1, C2 z) {
      __stcg(reinterpret_cast<float4*>(slot + (size_t)k1 * M + n2), make_float4(z.x.x, z.y.x, z.x.y, z.y.y));
    };
    put(0, v[0]);
    C2 w[CR];
    w[1] = C2{make_float2(t.x, t.z), make_float2(t.y, t.w)};
#pragma unroll
    for (int k1 = 2; k1 < CR; ++k1) w[k1] = (k1 % 2 == 0) ? c2mul(w[k1 / 2], w[k1 / 2]) : c2mul(w[k1 - 1], w[1]);
#pragma unroll
    for (int k1 = 1; k1 < CR; ++k1) put(k1, c2mul(v[k1], w[k1]));
  }
}

// Elements i, i + 1 into a 16-byte aligned row of device memory.
struct RowOutPairs {
  float2* row;
  SPX_DEV void operator()(uint32_t i, C2 z) const {
    __stcg(reinterpret_cast<float4*>(row + i), make_float4(z.x.x, z.y.x, z.x.y, z.y.y));
  }
};

}  // namespace spx
