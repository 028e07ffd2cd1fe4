// Register DFTs of 2 to 32 points, natural order in and out, unnormalised;
// inv = false: exp(-2 pi i m k / R).  Powers of two are radix-4 forms; other
// composite lengths are one Cooley-Tukey step over two smaller codelets with
// compile-time twiddles; odd primes fold the inputs into sums and differences
// of mirrored pairs, so that each output pair costs ((R-1)/2) real-by-complex
// multiply-adds of each kind instead of R - 1 complex ones.
#pragma once

#include "pg_common.cuh"

namespace pg {
namespace dft_detail {

// sin and cos of 2 pi m / R at compile time: the series of sin(x) and cos(x)
// on |x| <= pi / 4, every angle reduced to that octant by symmetry.
constexpr double series_sin(double x) {
  double t = x, s = x;
  for (int i = 1; i < 14; ++i) {
    t *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
    s += t;
  }
  return s;
}
constexpr double series_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int i = 1; i < 14; ++i) {
    t *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
    s += t;
  }
  return s;
}
constexpr double kTwoPi = 6.283185307179586476925286766559;
// cos(2 pi m / R): 8 m / R octants.
constexpr double unit_cos(int m, int R) {
  m %= R;
  if (m < 0) m += R;
  if (2 * m > R) m = R - m;                              // cos is even: angle in [0, pi]
  const bool neg = 4 * m > R;                            // past pi / 2
  const double q = neg ? 0.5 * R - m : (double)m;        // mirrored into [0, pi / 2]
  const double v = 8.0 * q <= R ? series_cos(kTwoPi * q / R) : series_sin(kTwoPi * (0.25 * R - q) / R);
  return neg ? -v : v;
}
constexpr double unit_sin(int m, int R) { return unit_cos(4 * m - R, 4 * R); }   // sin a = cos(a - pi / 2)

template <int R>
struct UnitTable {
  float c[R], s[R];
};
template <int R>
constexpr UnitTable<R> make_unit_table() {
  UnitTable<R> t{};
  for (int m = 0; m < R; ++m) {
    t.c[m] = (float)unit_cos(m, R);
    t.s[m] = (float)unit_sin(m, R);
  }
  return t;
}
template <int R>
__device__ constexpr UnitTable<R> kUnit = make_unit_table<R>();

}  // namespace dft_detail

__device__ __forceinline__ float2 twiddle(float2 v, float2 w, bool inv) {
  const float wy = inv ? -w.y : w.y;
  return make_float2(v.x * w.x - v.y * wy, v.x * wy + v.y * w.x);
}

__device__ __forceinline__ void dft2(float2& a, float2& b) {
  const float2 t = a;
  a = make_float2(t.x + b.x, t.y + b.y);
  b = make_float2(t.x - b.x, t.y - b.y);
}

__device__ __forceinline__ void dft4(float2& v0, float2& v1, float2& v2, float2& v3, bool inv) {
  const float2 t0 = make_float2(v0.x + v2.x, v0.y + v2.y), t1 = make_float2(v0.x - v2.x, v0.y - v2.y);
  const float2 t2 = make_float2(v1.x + v3.x, v1.y + v3.y), t3 = make_float2(v1.x - v3.x, v1.y - v3.y);
  // -i*t3 = (t3.y, -t3.x)
  const float2 m3 = inv ? make_float2(-t3.y, t3.x) : make_float2(t3.y, -t3.x);
  v0 = make_float2(t0.x + t2.x, t0.y + t2.y);
  v1 = make_float2(t1.x + m3.x, t1.y + m3.y);
  v2 = make_float2(t0.x - t2.x, t0.y - t2.y);
  v3 = make_float2(t1.x - m3.x, t1.y - m3.y);
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R], bool inv);

// R = A * B: m = B m1 + m2, k = k1 + A k2.
template <int A, int B>
__device__ __forceinline__ void dft_composite(float2 (&v)[A * B], bool inv) {
  constexpr int R = A * B;
#pragma unroll
  for (int m2 = 0; m2 < B; ++m2) {
    float2 u[A];
#pragma unroll
    for (int m1 = 0; m1 < A; ++m1) u[m1] = v[B * m1 + m2];
    dft<A>(u, inv);
    v[m2] = u[0];
#pragma unroll
    for (int k1 = 1; k1 < A; ++k1)
      v[B * k1 + m2] = m2 == 0 ? u[k1]
                               : twiddle(u[k1], make_float2(dft_detail::kUnit<R>.c[m2 * k1 % R],
                                                            -dft_detail::kUnit<R>.s[m2 * k1 % R]), inv);
  }
  float2 y[R];
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    float2 u[B];
#pragma unroll
    for (int m2 = 0; m2 < B; ++m2) u[m2] = v[B * k1 + m2];
    dft<B>(u, inv);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) y[k1 + A * k2] = u[k2];
  }
#pragma unroll
  for (int i = 0; i < R; ++i) v[i] = y[i];
}

// Odd prime R: X[k], X[R - k] = v0 + sum_j cos(2 pi j k / R) (v_j + v_{R-j})
//                               -/+ i sum_j sin(2 pi j k / R) (v_j - v_{R-j}).
template <int R>
__device__ __forceinline__ void dft_prime(float2 (&v)[R], bool inv) {
  constexpr int H = (R - 1) / 2;
  float2 a[H], b[H];
  const float2 v0 = v[0];
  float2 sum = v0;
#pragma unroll
  for (int j = 1; j <= H; ++j) {
    const float2 p = v[j], q = v[R - j];
    a[j - 1] = make_float2(p.x + q.x, p.y + q.y);
    b[j - 1] = make_float2(p.x - q.x, p.y - q.y);
    sum.x += a[j - 1].x;
    sum.y += a[j - 1].y;
  }
  v[0] = sum;
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    float2 e = v0, o = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      const float c = dft_detail::kUnit<R>.c[j * k % R], s = dft_detail::kUnit<R>.s[j * k % R];
      e.x += c * a[j - 1].x;
      e.y += c * a[j - 1].y;
      o.x += s * b[j - 1].x;
      o.y += s * b[j - 1].y;
    }
    // -i o = (o.y, -o.x)
    const float2 r = inv ? make_float2(-o.y, o.x) : make_float2(o.y, -o.x);
    v[k] = make_float2(e.x + r.x, e.y + r.y);
    v[R - k] = make_float2(e.x - r.x, e.y - r.y);
  }
}

// The larger power-of-two factor first, then the smallest odd one.
__host__ __device__ constexpr int dft_first_factor(int R) {
  if (R % 8 == 0 && R != 8) return 8;
  if (R % 4 == 0 && R != 4) return 4;
  if (R % 2 == 0 && R != 2) return 2;
  for (int p = 3; p * p <= R; p += 2)
    if (R % p == 0) return p;
  return 1;
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R], bool inv) {
  if constexpr (R == 1) {
    return;
  } else if constexpr (R == 2) {
    dft2(v[0], v[1]);
  } else if constexpr (R == 4) {
    dft4(v[0], v[1], v[2], v[3], inv);
  } else if constexpr (R == 16) {
    dft_composite<4, 4>(v, inv);
  } else {
    constexpr int A = dft_first_factor(R);
    if constexpr (A == 1) dft_prime<R>(v, inv);
    else dft_composite<A, R / A>(v, inv);
  }
}

}  // namespace pg
