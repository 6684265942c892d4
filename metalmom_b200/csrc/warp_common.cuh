// Device helpers shared by the frame-pair and tensor-core frame kernels:
// compile-time roots of unity, the quarter-table root lookup, stage-2 column
// assignment.
#pragma once
#include <math.h>

#include <type_traits>

#include "fft_radix.cuh"
#include "frame_common.cuh"

namespace mm {

// ---------------------------------------------------------------------------
// compile-time cos / sin of 2 pi k / d: octant reduction, then Taylor series
// in double (|x| <= pi/4, 12 terms: error far below float rounding)
// ---------------------------------------------------------------------------
constexpr double kPiD = 3.14159265358979323846264338327950288;

__host__ __device__ constexpr double ce_sin_q(double x) {
  double term = x, sum = x;
  for (int n = 1; n < 12; n++) {
    term *= -x * x / (double)((2 * n) * (2 * n + 1));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double ce_cos_q(double x) {
  double term = 1.0, sum = 1.0;
  for (int n = 1; n < 12; n++) {
    term *= -x * x / (double)((2 * n - 1) * (2 * n));
    sum += term;
  }
  return sum;
}
// which = 0: cos(2 pi k / d), 1: sin(2 pi k / d)
__host__ __device__ constexpr double ce_trig(long long k, long long d, int which) {
  k %= d;
  if (k < 0) k += d;
  const long long q = (8 * k) / d;                                   // octant 0..7
  const double phi = kPiD * (double)(8 * k - q * d) / (4.0 * (double)d);  // in [0, pi/4)
  const double psi = kPiD * (double)(d * (q + 1) - 8 * k) / (4.0 * (double)d);  // pi/4 - phi
  double c = 0.0, s = 0.0;
  switch (q) {
    case 0: c = ce_cos_q(phi); s = ce_sin_q(phi); break;
    case 1: c = ce_sin_q(psi); s = ce_cos_q(psi); break;
    case 2: c = -ce_sin_q(phi); s = ce_cos_q(phi); break;
    case 3: c = -ce_cos_q(psi); s = ce_sin_q(psi); break;
    case 4: c = -ce_cos_q(phi); s = -ce_sin_q(phi); break;
    case 5: c = -ce_sin_q(psi); s = -ce_cos_q(psi); break;
    case 6: c = ce_sin_q(phi); s = -ce_cos_q(phi); break;
    default: c = ce_cos_q(psi); s = -ce_sin_q(psi); break;
  }
  return which == 0 ? c : s;
}

template <int I, int N, typename Fn>
__device__ __forceinline__ void static_for(Fn &&fn) {
  if constexpr (I < N) {
    fn(std::integral_constant<int, I>{});
    static_for<I + 1, N>(fn);
  }
}

// a * exp(-2 pi i K / D), with the exact special angles spelled out.
template <int K, int D>
__device__ __forceinline__ cpx tw_const(cpx a) {
  constexpr int k = ((K % D) + D) % D;
  if constexpr (k == 0) {
    return a;
  } else if constexpr (4 * k == D) {
    return mul_mi(a);
  } else if constexpr (2 * k == D) {
    return {-a.x, -a.y};
  } else if constexpr (4 * k == 3 * D) {
    return mul_pi(a);
  } else if constexpr (8 * k == D) {
    return mul_w8_1(a);
  } else if constexpr (8 * k == 3 * D) {
    return mul_w8_3(a);
  } else if constexpr (8 * k == 5 * D) {
    return {-kR * (a.x + a.y), kR * (a.x - a.y)};
  } else if constexpr (8 * k == 7 * D) {
    return {kR * (a.x - a.y), kR * (a.x + a.y)};
  } else {
    constexpr float c = (float)ce_trig(k, D, 0);
    constexpr float s = -(float)ce_trig(k, D, 1);
    return {fmaf(a.x, c, -a.y * s), fmaf(a.x, s, a.y * c)};
  }
}

// W_N^s for any s >= 0 from the quarter table q[t] = W_N^t, t < N/4.
__device__ __forceinline__ cpx root_q(const float2 *q, int s, int N) {
  s &= N - 1;
  const int quarter = N >> 2;
  const int h = s / quarter, r = s - h * quarter;
  const float2 w = __ldg(q + r);
  switch (h) {
    case 0: return {w.x, w.y};
    case 1: return {w.y, -w.x};   // * (-i)
    case 2: return {-w.x, -w.y};  // * (-1)
    default: return {-w.y, w.x};  // * (+i)
  }
}

// Stage-2 column of slot c for lane l: columns k1 and 32 - k1 sit in one lane.
template <int TPF, int C, int c>
__device__ __forceinline__ int stage2_col(int l) {
  if constexpr (C == 1) {
    return l;
  } else if constexpr (c < C / 2) {
    return l + TPF * c;
  } else if constexpr (c == C / 2) {
    return l == 0 ? 16 : 32 - l;
  } else {
    return 32 - l - TPF * (c - C / 2);
  }
}

}  // namespace mm
