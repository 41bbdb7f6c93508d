// Small in-register DFTs of compile-time length: the steps of the line
// transforms (local_lines.cuh).  Lengths 2..16 run fully unrolled: coprime
// composite lengths (6, 10, 12, 15) by the prime-factor mapping, 8, 9 and 16
// by the Cooley-Tukey split.  Every multiply-add is an explicit fma, so that
// a length gives the same bits in every kernel that uses it.
#pragma once

#include <type_traits>

#include "qeb_common.cuh"

namespace qeb {

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

// a + s b (s real)
template <typename T>
__device__ __forceinline__ C2<T> add_scaled(C2<T> a, T s, C2<T> b) {
  return mk<T>(fma_t(s, b.re, a.re), fma_t(s, b.im, a.im));
}
// a + i s b (s real)
template <typename T>
__device__ __forceinline__ C2<T> add_scaled_i(C2<T> a, T s, C2<T> b) {
  return mk<T>(fma_t(-s, b.im, a.re), fma_t(s, b.re, a.im));
}
// a + i b or a - i b
template <typename T, bool PLUS>
__device__ __forceinline__ C2<T> add_i(C2<T> a, C2<T> b) {
  return PLUS ? mk<T>(a.re - b.im, a.im + b.re) : mk<T>(a.re + b.im, a.im - b.re);
}
// a w and a conj(w)
template <typename T>
__device__ __forceinline__ C2<T> twiddle(C2<T> a, C2<T> w) {
  return mk<T>(fma_t(a.re, w.re, -(a.im * w.im)), fma_t(a.re, w.im, a.im * w.re));
}
template <typename T>
__device__ __forceinline__ C2<T> twiddle_conj(C2<T> a, C2<T> w) {
  return mk<T>(fma_t(a.re, w.re, a.im * w.im), fma_t(a.im, w.re, -(a.re * w.im)));
}

template <int N> struct Split { static constexpr int A = 1, B = N; };
template <> struct Split<6> { static constexpr int A = 2, B = 3; };
template <> struct Split<9> { static constexpr int A = 3, B = 3; };
template <> struct Split<10> { static constexpr int A = 2, B = 5; };
template <> struct Split<12> { static constexpr int A = 3, B = 4; };
template <> struct Split<15> { static constexpr int A = 3, B = 5; };
template <> struct Split<16> { static constexpr int A = 4, B = 4; };

constexpr int gcd_c(int a, int b) { return b == 0 ? a : gcd_c(b, a % b); }

// The inverse of a modulo m (a and m coprime, both small).
constexpr int inverse_mod_c(int a, int m) {
  for (int x = 1; x < m; ++x)
    if ((a * x) % m == 1) return x;
  return m == 1 ? 0 : -1;
}

// exp(-2 pi i m / N) of the non-coprime splits (N = 9: m = 1, 2, 4;
// N = 16: m = 1, 2, 3, 4, 6, 9), rounded once to T.
template <typename T, int N>
__device__ __forceinline__ C2<T> root(int m) {
  constexpr double c9[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5,
                            -0.93969262078590838405};
  constexpr double s9[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937,
                            0.86602540378443864676, 0.34202014332566873304};
  constexpr double c16[10] = {1.0, 0.92387953251128675613, 0.70710678118654752440,
                              0.38268343236508977173, 0.0, -0.38268343236508977173,
                              -0.70710678118654752440, -0.92387953251128675613, -1.0,
                              -0.92387953251128675613};
  constexpr double s16[10] = {0.0, 0.38268343236508977173, 0.70710678118654752440,
                              0.92387953251128675613, 1.0, 0.92387953251128675613,
                              0.70710678118654752440, 0.38268343236508977173, 0.0,
                              -0.38268343236508977173};
  return N == 9 ? mk<T>((T)c9[m % 5], (T)-s9[m % 5]) : mk<T>((T)c16[m % 10], (T)-s16[m % 10]);
}

// Known-zero mask of the inputs u[n1] = v[(stride n1 + offset) mod N], n1 < A,
// from the mask Z of v.
template <int A, int N, unsigned Z, int STRIDE, int OFFSET>
constexpr unsigned sub_zero_mask() {
  unsigned m = 0;
  for (int n1 = 0; n1 < A; ++n1)
    if ((Z >> ((STRIDE * n1 + OFFSET) % N)) & 1u) m |= 1u << n1;
  return m;
}

// Calls fn(std::integral_constant<int, I>{}) for I = BEGIN .. END - 1.
template <int BEGIN, int END, class Fn>
__device__ __forceinline__ void static_for(Fn&& fn) {
  if constexpr (BEGIN < END) {
    fn(std::integral_constant<int, BEGIN>{});
    static_for<BEGIN + 1, END>(fn);
  }
}

// In-register DFT of compile-time length N (sign +1 if BWD else -1).
// Bit i of Z marks input i as zero: it is neither read nor added (the line
// transforms' blocks without sticks), otherwise the same operations.
// Coprime splits N = A B use the prime-factor (Good-Thomas) mapping: input
// n = (B n1 + A n2) mod N, output k with k = k1 (mod A) and k = k2 (mod B),
// so w_N^(n k) = w_A^(n1 k1) w_B^(n2 k2) and no twiddle multiplications sit
// between the two stages.
template <typename T, int N, bool BWD, unsigned Z = 0u>
__device__ __forceinline__ void dft(C2<T>* v) {
  constexpr T sgn = BWD ? T(1) : T(-1);
  constexpr unsigned kAll = (1u << N) - 1u;
  if constexpr (N == 1) {
    return;
  } else if constexpr ((Z & kAll) == kAll) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = mk<T>(0, 0);
  } else if constexpr ((Z & kAll) == (kAll & ~1u)) {  // only v[0]: every output is v[0]
#pragma unroll
    for (int i = 1; i < N; ++i) v[i] = v[0];
  } else if constexpr (N == 2) {
    if constexpr (Z & 1u) {  // (0, b) -> (b, -b)
      v[0] = v[1];
      v[1] = mk<T>(-v[1].re, -v[1].im);
    } else {
      const C2<T> a = v[0], b = v[1];
      v[0] = a + b;
      v[1] = a - b;
    }
  } else if constexpr (N == 3 && Z == 3u) {  // only v[2]
    const C2<T> c = v[2], m = scale(c, T(-0.5));
    v[0] = c;
    v[1] = add_scaled_i(m, -sgn * T(kSin60), c);
    v[2] = add_scaled_i(m, sgn * T(kSin60), c);
  } else if constexpr (N == 3 && Z == 5u) {  // only v[1]
    const C2<T> b = v[1], m = scale(b, T(-0.5));
    v[0] = b;
    v[1] = add_scaled_i(m, sgn * T(kSin60), b);
    v[2] = add_scaled_i(m, -sgn * T(kSin60), b);
  } else if constexpr (N == 3) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if ((Z >> i) & 1u) v[i] = mk<T>(0, 0);
    const C2<T> s = v[1] + v[2], d = v[1] - v[2];
    const C2<T> m = add_scaled(v[0], T(-0.5), s);
    v[0] = v[0] + s;
    v[1] = add_scaled_i(m, sgn * T(kSin60), d);
    v[2] = add_scaled_i(m, -sgn * T(kSin60), d);
  } else if constexpr (N == 4) {
    C2<T> e[2] = {v[0], v[2]}, o[2] = {v[1], v[3]};
    dft<T, 2, BWD, sub_zero_mask<2, 4, Z, 2, 0>()>(e);
    dft<T, 2, BWD, sub_zero_mask<2, 4, Z, 2, 1>()>(o);
    v[0] = e[0] + o[0];
    v[2] = e[0] - o[0];
    v[1] = add_i<T, BWD>(e[1], o[1]);
    v[3] = add_i<T, !BWD>(e[1], o[1]);
  } else if constexpr (N == 5) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if ((Z >> i) & 1u) v[i] = mk<T>(0, 0);
    const C2<T> a = v[0];
    const C2<T> s1 = v[1] + v[4], d1 = v[1] - v[4], s2 = v[2] + v[3], d2 = v[2] - v[3];
    v[0] = a + s1 + s2;
    const C2<T> m1 = add_scaled(add_scaled(a, T(kCos72), s1), T(kCos144), s2);
    const C2<T> m2 = add_scaled(add_scaled(a, T(kCos144), s1), T(kCos72), s2);
    const C2<T> p1 = add_scaled(scale(d2, T(kSin144)), T(kSin72), d1);
    const C2<T> p2 = add_scaled(scale(d2, T(-kSin72)), T(kSin144), d1);
    v[1] = add_i<T, BWD>(m1, p1);
    v[4] = add_i<T, !BWD>(m1, p1);
    v[2] = add_i<T, BWD>(m2, p2);
    v[3] = add_i<T, !BWD>(m2, p2);
  } else if constexpr (N == 8) {
    // two length-4 DFTs (even and odd inputs), then w8^k = ((1 +- i)/sqrt 2)^k
    // folded into the last additions as fma
    constexpr T r = T(0.70710678118654752440084436210484903928L);
    C2<T> e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft<T, 4, BWD, sub_zero_mask<4, 8, Z, 2, 0>()>(e);
    dft<T, 4, BWD, sub_zero_mask<4, 8, Z, 2, 1>()>(o);
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    v[2] = add_i<T, BWD>(e[2], o[2]);
    v[6] = add_i<T, !BWD>(e[2], o[2]);
    const C2<T> p = add_i<T, BWD>(o[1], o[1]);    // (1 + sgn i) o1
    const C2<T> q = add_i<T, !BWD>(o[3], o[3]);   // (1 - sgn i) o3
    v[1] = add_scaled(e[1], r, p);
    v[5] = add_scaled(e[1], -r, p);
    v[3] = add_scaled(e[3], -r, q);               // w8^3 = -(1 - sgn i)/sqrt 2
    v[7] = add_scaled(e[3], r, q);
  } else if constexpr (gcd_c(Split<N>::A, Split<N>::B) == 1) {
    constexpr int A = Split<N>::A, B = Split<N>::B;
    constexpr int eA = B * inverse_mod_c(B % A, A), eB = A * inverse_mod_c(A % B, B);
    static_assert(eA % A == 1 && eA % B == 0 && eB % B == 1 && eB % A == 0,
                  "CRT idempotents of the prime-factor split");
    C2<T> y[A][B];
    static_for<0, B>([&](auto c) {
      constexpr int n2 = decltype(c)::value;
      C2<T> u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) u[n1] = v[(B * n1 + A * n2) % N];
      dft<T, A, BWD, sub_zero_mask<A, N, Z, B, A * n2>()>(u);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) y[k1][n2] = u[k1];
    });
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      dft<T, B, BWD>(y[k1]);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[(k1 * eA + k2 * eB) % N] = y[k1][k2];
    }
  } else {
    constexpr int A = Split<N>::A, B = Split<N>::B;
    C2<T> y[B][A];
    static_for<0, B>([&](auto c) {
      constexpr int n2 = decltype(c)::value;
      C2<T> u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) u[n1] = v[B * n1 + n2];
      dft<T, A, BWD, sub_zero_mask<A, N, Z, B, n2>()>(u);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) {
        if (n2 * k1 == 0)
          y[n2][k1] = u[k1];
        else
          y[n2][k1] = BWD ? twiddle_conj(u[k1], root<T, N>(n2 * k1))
                          : twiddle(u[k1], root<T, N>(n2 * k1));
      }
    });
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      C2<T> w[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) w[n2] = y[n2][k1];
      dft<T, B, BWD>(w);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = w[k2];
    }
  }
}

}  // namespace qeb
