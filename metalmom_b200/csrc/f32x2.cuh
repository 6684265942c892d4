// Two float32 lanes in one 64-bit register (sm_100a packed arithmetic) and the
// register DFTs over them: lane 0 and lane 1 belong to two frames, so every
// butterfly, twiddle and product below serves both frames in one instruction.
//
// Measured on B200 (warp instructions per clock and SM, 8 to 16 resident
// warps): fma / add / mul.f32x2 1.9-2.0, scalar fma 3.3, i.e. up to the same
// 128 float32 lanes with half the issue slots.  A broadcast scalar operand, a
// compile-time constant pair and a negated operand cost no instruction of
// their own (warp-instruction counts of a probe with and without them).
#pragma once
#include <cuda_runtime.h>

#include "warp_common.cuh"

namespace mm {

struct f2 {
  unsigned long long v;
};

__device__ __forceinline__ f2 pk2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 dup2(float a) { return pk2(a, a); }
__device__ __forceinline__ void un2(f2 a, float &x, float &y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ float lo2(f2 a) {
  float x, y;
  un2(a, x, y);
  return x;
}
__device__ __forceinline__ float hi2(f2 a) {
  float x, y;
  un2(a, x, y);
  return y;
}
__device__ __forceinline__ f2 neg2(f2 a) {
  float x, y;
  un2(a, x, y);
  return pk2(-x, -y);
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 sel2(bool p, f2 a, f2 b) {
  f2 r;
  r.v = p ? a.v : b.v;
  return r;
}
__device__ __forceinline__ f2 shfl2(f2 a, int src) {
  float x, y;
  un2(a, x, y);
  return pk2(__shfl_sync(0xffffffffu, x, src), __shfl_sync(0xffffffffu, y, src));
}

// One complex point of both frames.
struct cpx2 {
  f2 x, y;
};

__device__ __forceinline__ cpx2 cadd(cpx2 a, cpx2 b) { return {add2(a.x, b.x), add2(a.y, b.y)}; }
__device__ __forceinline__ cpx2 csub(cpx2 a, cpx2 b) { return {sub2(a.x, b.x), sub2(a.y, b.y)}; }
__device__ __forceinline__ cpx2 csel(bool p, cpx2 a, cpx2 b) { return {sel2(p, a.x, b.x), sel2(p, a.y, b.y)}; }
// a * w, the same w for both frames
__device__ __forceinline__ cpx2 cmul(cpx2 a, cpx w) {
  const f2 wx = dup2(w.x), wy = dup2(w.y);
  return {fma2(a.x, wx, neg2(mul2(a.y, wy))), fma2(a.x, wy, mul2(a.y, wx))};
}

// W = exp(-2 pi i K / D) factored as W a = scale * rot(a), the larger of |cos|
// and |sin| as the scale and a ratio of at most 1 inside rot: rot takes two
// FMAs and the scale rides in the FMAs of the butterfly that follows (6
// operations for e +- W o instead of 8).
template <int K, int D>
struct Rot {
  static constexpr int k = ((K % D) + D) % D;
  static constexpr float c = (4 * k == D || 4 * k == 3 * D) ? 0.0f : (float)ce_trig(k, D, 0);
  static constexpr float s = (k == 0 || 2 * k == D) ? 0.0f : (float)ce_trig(k, D, 1);
  static constexpr bool cform = (c < 0 ? -c : c) >= (s < 0 ? -s : s);
  static constexpr float scale = cform ? c : s;
  static constexpr float ratio = cform ? (float)(ce_trig(k, D, 1) / ce_trig(k, D, 0))
                                       : (float)(ce_trig(k, D, 0) / ce_trig(k, D, 1));
  // special ratios are exact: 0 (multiples of a quarter turn), +-1 (odd eighths)
  static constexpr int kind = (4 * k) % D == 0 ? 0 : ((8 * k) % D == 0 ? 1 : 2);
  static constexpr float rt = kind == 1 ? (ratio > 0 ? 1.0f : -1.0f) : ratio;
  static __device__ __forceinline__ cpx2 rot(cpx2 a) {
    if constexpr (cform) {  // (x + r y, y - r x)
      if constexpr (kind == 0) return a;
      else if constexpr (kind == 1 && rt > 0) return {add2(a.x, a.y), sub2(a.y, a.x)};
      else if constexpr (kind == 1) return {sub2(a.x, a.y), add2(a.y, a.x)};
      else return {fma2(a.y, dup2(rt), a.x), fma2(a.x, dup2(-rt), a.y)};
    } else {  // (r x + y, r y - x)
      if constexpr (kind == 0) return {a.y, neg2(a.x)};
      else return {fma2(a.x, dup2(rt), a.y), fma2(a.y, dup2(rt), neg2(a.x))};
    }
  }
};
// e + S r and e - S r for a compile-time S
template <typename R>
__device__ __forceinline__ void rot_butterfly(cpx2 e, cpx2 r, cpx2 &lo, cpx2 &hi) {
  if constexpr (R::scale == 1.0f) {
    lo = cadd(e, r);
    hi = csub(e, r);
  } else if constexpr (R::scale == -1.0f) {
    lo = csub(e, r);
    hi = cadd(e, r);
  } else {
    const f2 p = dup2(R::scale), n = dup2(-R::scale);
    lo = {fma2(r.x, p, e.x), fma2(r.y, p, e.y)};
    hi = {fma2(r.x, n, e.x), fma2(r.y, n, e.y)};
  }
}

// In-place 4-point DFT, natural order.
__device__ __forceinline__ void dft4(cpx2 &a0, cpx2 &a1, cpx2 &a2, cpx2 &a3) {
  const cpx2 t0 = cadd(a0, a2), t1 = csub(a0, a2);
  const cpx2 t2 = cadd(a1, a3), t3 = csub(a1, a3);
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = {add2(t1.x, t3.y), sub2(t1.y, t3.x)};
  a3 = {sub2(t1.x, t3.y), add2(t1.y, t3.x)};
}

// 4-point DFT of (a0, W^K a1, W^2K a2, W^3K a3), W = exp(-2 pi i / D), the
// twiddles folded into the butterflies (Rot): 22 operations instead of 28.
template <int K, int D>
__device__ __forceinline__ void dft4_tw(cpx2 &a0, cpx2 &a1, cpx2 &a2, cpx2 &a3) {
  using R1 = Rot<K, D>;
  using R2 = Rot<2 * K, D>;
  using R3 = Rot<3 * K, D>;
  // the odd inputs' common scale, up to sign
  static_assert(R3::scale == R1::scale || R3::scale == -R1::scale, "odd twiddles share their scale");
  cpx2 t0, t1;
  rot_butterfly<R2>(a0, R2::rot(a2), t0, t1);
  const cpx2 r1 = R1::rot(a1), r3 = R3::rot(a3);
  cpx2 t2, t3;
  if constexpr (R3::scale == R1::scale) {
    t2 = cadd(r1, r3);
    t3 = csub(r1, r3);
  } else {
    t2 = csub(r1, r3);
    t3 = cadd(r1, r3);
  }
  rot_butterfly<R1>(t0, t2, a0, a2);
  rot_butterfly<R1>(t1, {t3.y, neg2(t3.x)}, a1, a3);
}

// In-place 8-point DFT, natural order: 4-point DFTs of the even and odd
// points, then the radix-2 combine with W_8 folded in.
__device__ __forceinline__ void dft8(cpx2 *v) {
  dft4(v[0], v[2], v[4], v[6]);
  dft4(v[1], v[3], v[5], v[7]);
  cpx2 o[8];
  static_for<0, 4>([&](auto ki) {
    constexpr int k = decltype(ki)::value;
    using R = Rot<k, 8>;
    rot_butterfly<R>(v[2 * k], R::rot(v[2 * k + 1]), o[k], o[k + 4]);
  });
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = o[i];
}

// In-place 16-point DFT, natural order (n = 4 n1 + n2, k = k1 + 4 k2).
__device__ __forceinline__ void dft16(cpx2 *v) {
#pragma unroll
  for (int n2 = 0; n2 < 4; n2++) dft4(v[n2], v[n2 + 4], v[n2 + 8], v[n2 + 12]);
  dft4(v[0], v[1], v[2], v[3]);
  dft4_tw<1, 16>(v[4], v[5], v[6], v[7]);
  dft4_tw<2, 16>(v[8], v[9], v[10], v[11]);
  dft4_tw<3, 16>(v[12], v[13], v[14], v[15]);
  cpx2 o[16];
#pragma unroll
  for (int k1 = 0; k1 < 4; k1++)
#pragma unroll
    for (int k2 = 0; k2 < 4; k2++) o[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = o[i];
}

// In-place 32-point DFT, natural order: radix-2 over two 16-point DFTs (380
// operations, 444 with separate twiddle products).
__device__ __forceinline__ void dft32(cpx2 *v) {
  cpx2 e[16], o[16];
#pragma unroll
  for (int m = 0; m < 16; m++) {
    e[m] = v[2 * m];
    o[m] = v[2 * m + 1];
  }
  dft16(e);
  dft16(o);
  static_for<0, 16>([&](auto ki) {
    constexpr int k = decltype(ki)::value;
    using R = Rot<k, 32>;
    rot_butterfly<R>(e[k], R::rot(o[k]), v[k], v[k + 16]);
  });
}

template <int R>
__device__ __forceinline__ void dft_any(cpx2 *v) {
  if constexpr (R == 32) dft32(v);
  else if constexpr (R == 16) dft16(v);
  else if constexpr (R == 8) dft8(v);
  else {
    static_assert(R == 4, "radix must be 4, 8, 16 or 32");
    dft4(v[0], v[1], v[2], v[3]);
  }
}

}  // namespace mm
