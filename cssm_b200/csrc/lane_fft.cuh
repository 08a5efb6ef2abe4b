// N-point complex FFT of one lane, in registers, for any N that fits there: natural order in and out, e^{-...}, unscaled.
//
// Sizes with two coprime factors are split by the prime-factor mapping (Good 1958, Thomas 1963: an N1 x N2 transform without
// twiddles, the orders in and out are compile-time index maps and cost nothing), powers of a prime by Cooley and Tukey's; odd primes are
// direct, the terms j and R - j together (half the multiplications).  Everything is unrolled, so the constants are immediates.
// 56 points: 8 transforms of 7, 7 of 8, about 1070 operations, 146 registers a lane.
// Scalar adds and multiply-adds: packed ones are as fast (geometric mean over 44 sides of gated_spectral_fft 0.99 of the scalar form's speed).
#pragma once
#include "common.cuh"

namespace cssm {

constexpr double LANE_PI = 3.14159265358979323846264338327950288;
// sin and cos of 2 pi p / n by their Taylor series within an eighth of a turn
__host__ __device__ constexpr double lane_taylor_sin(double a) {
  double t = a, s = a;
  for (int i = 1; i < 12; ++i) { t *= -a * a / ((2 * i) * (2 * i + 1)); s += t; }
  return s;
}
__host__ __device__ constexpr double lane_taylor_cos(double a) {
  double t = 1, s = 1;
  for (int i = 1; i < 12; ++i) { t *= -a * a / ((2 * i - 1) * (2 * i)); s += t; }
  return s;
}
__host__ __device__ constexpr double cos_turn(int p, int n) {
  p %= n;
  if (2 * p > n) p = n - p;
  const bool neg = 4 * p > n;
  const int q = neg ? n - 2 * p : 2 * p;
  const double a = LANE_PI * q / n;
  const double v = 4 * q > n ? lane_taylor_sin(LANE_PI * (n - 2 * q) / (2.0 * n)) : lane_taylor_cos(a);
  return neg ? -v : v;
}
__host__ __device__ constexpr double sin_turn(int p, int n) { return cos_turn(4 * (p % n) + 3 * n, 4 * n); }

template <int N> struct LaneTurn { float c[N], s[N]; };
template <int N> __host__ __device__ constexpr LaneTurn<N> lane_turns() {
  LaneTurn<N> t{};
  for (int p = 0; p < N; ++p) { t.c[p] = (float)cos_turn(p, N); t.s[p] = (float)sin_turn(p, N); }
  return t;
}
// a + c b, c b: real c
__device__ __forceinline__ cf lane_fma(float c, cf b, cf a) { return mk(fmaf(c, b.x, a.x), fmaf(c, b.y, a.y)); }
__device__ __forceinline__ cf lane_mul(float c, cf b) { return mk(c * b.x, c * b.y); }

__host__ __device__ constexpr int lane_prime_power(int n) {       // largest power of the smallest prime in n
  int p = 2;
  while (n % p) ++p;
  int q = 1;
  while (n % p == 0) { n /= p; q *= p; }
  return q;
}
__host__ __device__ constexpr bool lane_is_prime(int n) { for (int p = 2; p * p <= n; ++p) if (n % p == 0) return false; return n > 1; }
__host__ __device__ constexpr int lane_inverse(int a, int m) { for (int i = 1; i < m; ++i) if (a * i % m == 1) return i; return m == 1 ? 0 : -1; }
__host__ __device__ constexpr int lane_radix(int n) { return n % 2 == 0 ? 4 : n % 7 == 0 ? 7 : n % 5 == 0 ? 5 : 3; }

template <int N> __device__ __forceinline__ void lane_dft(cf (&x)[N]);

template <int R> __device__ __forceinline__ void lane_dft_odd(cf (&x)[R]) {
  constexpr LaneTurn<R> tw = lane_turns<R>();
  constexpr int M = R / 2;
  cf s[M], d[M];
#pragma unroll
  for (int j = 0; j < M; ++j) { s[j] = x[1 + j] + x[R - 1 - j]; d[j] = x[1 + j] - x[R - 1 - j]; }
  cf X0 = x[0];
#pragma unroll
  for (int j = 0; j < M; ++j) X0 = X0 + s[j];
  const cf x0 = x[0];
#pragma unroll
  for (int k = 1; k <= M; ++k) {
    cf a = x0, b = lane_mul(tw.s[k % R], d[0]);
#pragma unroll
    for (int j = 0; j < M; ++j) a = lane_fma(tw.c[(j + 1) * k % R], s[j], a);
#pragma unroll
    for (int j = 1; j < M; ++j) b = lane_fma(tw.s[(j + 1) * k % R], d[j], b);
    x[k] = mk(a.x + b.y, a.y - b.x);          // a - i b
    x[R - k] = mk(a.x - b.y, a.y + b.x);
  }
  x[0] = X0;
}

template <int N> __device__ __forceinline__ void lane_dft(cf (&x)[N]) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2) {
    const cf a = x[0], b = x[1];
    x[0] = a + b; x[1] = a - b;
  } else if constexpr (N == 4) {
    const cf s0 = x[0] + x[2], d0 = x[0] - x[2], s1 = x[1] + x[3], d1 = x[1] - x[3];
    x[0] = s0 + s1; x[2] = s0 - s1;
    x[1] = mk(d0.x + d1.y, d0.y - d1.x); x[3] = mk(d0.x - d1.y, d0.y + d1.x);
  } else if constexpr (N == 8) {
    constexpr float R = 0.70710678118654752440f;
    cf b0 = x[0] + x[4], b4 = x[0] - x[4];
    cf b1 = x[1] + x[5], b5 = x[1] - x[5];
    cf b2 = x[2] + x[6], b6 = x[2] - x[6];
    cf b3 = x[3] + x[7], b7 = x[3] - x[7];
    b5 = mk(R * (b5.x + b5.y), R * (b5.y - b5.x));
    b7 = mk(R * (b7.y - b7.x), -R * (b7.x + b7.y));
    cf c0 = b0 + b2, c2 = b0 - b2, c1 = b1 + b3, d3 = b1 - b3;
    cf c4 = mk(b4.x + b6.y, b4.y - b6.x), c6 = mk(b4.x - b6.y, b4.y + b6.x), c5 = b5 + b7, d7 = b5 - b7;
    x[0] = c0 + c1; x[4] = c0 - c1;
    x[2] = mk(c2.x + d3.y, c2.y - d3.x); x[6] = mk(c2.x - d3.y, c2.y + d3.x);
    x[1] = c4 + c5; x[5] = c4 - c5;
    x[3] = mk(c6.x + d7.y, c6.y - d7.x); x[7] = mk(c6.x - d7.y, c6.y + d7.x);
  } else if constexpr (lane_is_prime(N)) {
    lane_dft_odd<N>(x);
  } else if constexpr (lane_prime_power(N) != N) {
    // Good-Thomas: no twiddles
    constexpr int A = lane_prime_power(N), B = N / A;
    cf y[A][B];
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
      for (int b = 0; b < B; ++b) y[a][b] = x[(a * B + b * A) % N];
#pragma unroll
    for (int a = 0; a < A; ++a) lane_dft<B>(y[a]);
#pragma unroll
    for (int b = 0; b < B; ++b) {
      cf t[A];
#pragma unroll
      for (int a = 0; a < A; ++a) t[a] = y[a][b];
      lane_dft<A>(t);
#pragma unroll
      for (int a = 0; a < A; ++a) x[(a * B * lane_inverse(B % A, A) + b * A * lane_inverse(A % B, B)) % N] = t[a];
    }
  } else {
    constexpr int R = lane_radix(N), M = N / R;
    constexpr LaneTurn<N> tw = lane_turns<N>();
    cf y[R][M];
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int m = 0; m < M; ++m) y[r][m] = x[R * m + r];
      lane_dft<M>(y[r]);
#pragma unroll
      for (int m = 1; m < M; ++m) {
        const int p = r * m;
        if (p == 0) continue;
        const float c = tw.c[p], s = tw.s[p];
        const cf t = y[r][m];
        if (4 * p == N) y[r][m] = mk(t.y, -t.x);
        else y[r][m] = mk(t.x * c + t.y * s, t.y * c - t.x * s);
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
      cf t[R];
#pragma unroll
      for (int r = 0; r < R; ++r) t[r] = y[r][m];
      lane_dft<R>(t);
#pragma unroll
      for (int r = 0; r < R; ++r) x[m + M * r] = t[r];
    }
  }
}
}  // namespace cssm
