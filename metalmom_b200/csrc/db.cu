// dB scaling over a flat array (mm_power_to_db, mm_amplitude_to_db and their
// device-buffer forms; Scaling.swift:73-118): y = mult log10(max(x, amin) / ref),
// floored at max(y) - top_db when top_db > 0, ref given or max(x).
//
// For amin > 0 the largest y belongs to the largest max(x, amin), so the floor
// and a device-side ref need one pass over x for its maximum (4 bytes a value)
// and one that computes and writes y (8 bytes): 12 bytes a value where the
// three-pass form moved 20 (reference pass, log pass, floor pass in place).
// - db_small_kernel, up to 32 768 values: one CTA holds them in registers, so
//   both passes are one launch without scratch memory.
// - db_max_kernel + db_apply_kernel above: per-block maxima in scratch, which
//   every block of the second kernel reduces for itself; no slots to reset, no
//   atomics.  The second kernel walks x from its end, where the first one left
//   it in L2.
//
// The logarithm was what the second pass spent its time on (42.3 M values, 169
// MB, ref = max(x): 86 us where its 338 MB take 52), an IEEE division and a
// log10f a value.  Values whose quotient is surely a normal float32 now go two
// at a time in packed arithmetic (db_pair): the call 120 -> 106 us (the first
// pass takes 28 of it), its error against float64 3.7e-8 -> 2.0e-8.  Measured
// and left out: six resident blocks an SM instead of five (107 us), streaming
// stores (107 us).
//
// amin <= 0 (or NaN) keeps the pass-by-pass form: a logarithm of a negative
// number is NaN and the maximum must skip it.
#include <math.h>

#include "f32x2.cuh"
#include "frame_common.cuh"
#include "kernels.h"

namespace mm {

namespace {

constexpr int kDbThreads = 256;
constexpr int kDbSmallThreads = 1024;
constexpr int kDbSmallPer = 8;  // float4 per thread
constexpr long long kDbSmallMax = 4LL * kDbSmallPer * kDbSmallThreads;

__device__ __forceinline__ float db_value(float x, float mult, float amin, float ref) {
  return mult * log10f(vthr(x, amin) / ref);
}

// Block-wide {maximum, any NaN} of x's share; every thread gets it.
template <int THREADS>
__device__ __forceinline__ void block_max(float &vmax, bool &nan) {
  __shared__ float red[THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = vmax;
  nan = __syncthreads_or(nan) != 0;
  float v = (threadIdx.x & 31) < THREADS / 32 ? red[threadIdx.x & 31] : -INFINITY;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  vmax = v;
}

// What a launch's values have in common.
struct Levels {
  float mult, amin, ref, thr;  // thr: the floor (-inf: none)
  bool packed;                 // db_pair applies to values up to kPairHigh
  bool all;                    // ... and no value is larger
  float inv, twice;            // its 1 / ref, and mult / 10
};
// Range of db_pair: which form a value takes depends on it, amin and ref
// alone, so that every route gives it the same result.
constexpr float kPairLow = 8.67361737988403547e-19f, kPairHigh = 1.152921504606846976e18f;  // 2^-60, 2^60

// mult log10(x / ref) of two values where x, ref and so the quotient are well
// inside the normal range.
// - Quotient: with inv the correctly rounded 1 / ref, one residual step from
//   x inv gives the correctly rounded x / ref (Markstein, IBM J. Res. Dev. 34,
//   1990), the value that db_value takes the logarithm of.
// - Logarithm: x / ref = 2^e (1 + f) with 1 + f in [sqrt(1/2), sqrt(2)), and
//   10 log10(1 + f) = c f + f^2 Q(f), Q the weighted least-squares polynomial of degree 9
//   at Chebyshev points (its error: 1e-9 of the result).  c and 10 log10(2) are carried in two
//   floats, so the result is off by little more than its last rounding.
__device__ __forceinline__ f2 db_pair(f2 x, const Levels &lv) {
  const f2 inv = dup2(lv.inv);
  const f2 q0 = mul2(x, inv);
  const f2 q = fma2(fma2(neg2(q0), dup2(lv.ref), x), inv, q0);
  float qa, qb;
  un2(q, qa, qb);
  const int ia = __float_as_int(qa), ib = __float_as_int(qb);
  constexpr int kSqrtHalf = 0x3f3504f3, kBias = 0x4b400000;  // kBias: 1.5 2^23, to which e is added as an integer
  const int ta = ia - kSqrtHalf, tb = ib - kSqrtHalf;
  const f2 m = pk2(__int_as_float(ia - (ta & 0xff800000)), __int_as_float(ib - (tb & 0xff800000)));
  const f2 e = sub2(pk2(__int_as_float((ta >> 23) + kBias), __int_as_float((tb >> 23) + kBias)), dup2(12582912.0f));
  const f2 f = sub2(m, dup2(1.0f));
  constexpr float kQ[10] = {-2.1714723110198975f, 1.4476473331451416f,  -1.0857372283935547f, 0.8686825633049011f,
                            -0.7238692045211792f, 0.6175169944763184f,  -0.5388593673706055f, 0.5165238976478577f,
                            -0.5068863034248352f, 0.2925231456756592f};
  f2 g = dup2(kQ[9]);
#pragma unroll
  for (int i = 8; i >= 0; i--) g = fma2(g, f, dup2(kQ[i]));
  g = fma2(g, f, dup2(1.9699272335452558e-07f));  // 10 / ln 10 = 4.342944622039795 + this
  f2 y = fma2(f, dup2(4.342944622039795f), mul2(f, g));
  y = fma2(e, dup2(3.560404593372368e-08f), y);  // 10 log10(2) = 3.0102999210357666 + this
  y = fma2(e, dup2(3.0102999210357666f), y);
  return mul2(y, dup2(lv.twice));
}

__device__ __forceinline__ Levels levels(float mult, float amin, float ref) {
  Levels lv{mult, amin, ref, -INFINITY, false, false, 0.0f, 1.0f};
  lv.packed = amin >= kPairLow && amin <= kPairHigh && ref >= kPairLow && ref <= kPairHigh &&  // false for NaN
              (mult == 10.0f || mult == 20.0f);
  if (lv.packed) lv.inv = 1.0f / ref;
  if (mult == 20.0f) lv.twice = 2.0f;
  return lv;
}
// dB of two values
__device__ __forceinline__ void db_two(float &a, float &b, const Levels &lv) {
  const float xa = vthr(a, lv.amin), xb = vthr(b, lv.amin);
  if (lv.packed && (lv.all || fmaxf(xa, xb) <= kPairHigh)) {
    un2(db_pair(pk2(xa, xb), lv), a, b);
  } else {
    a = lv.packed && xa <= kPairHigh ? lo2(db_pair(dup2(xa), lv)) : db_value(a, lv.mult, lv.amin, lv.ref);
    b = lv.packed && xb <= kPairHigh ? lo2(db_pair(dup2(xb), lv)) : db_value(b, lv.mult, lv.amin, lv.ref);
  }
}
// The same with what follows from max(x) (NaNs skipped) and "x holds a NaN".
__device__ __forceinline__ Levels levels_of_max(float xmax, bool nan, float ref, bool ref_max, float mult, float amin,
                                                float top_db) {
  if (ref_max) ref = nan ? __int_as_float(0x7fc00000) : xmax;
  Levels lv = levels(mult, amin, ref);
  lv.all = lv.packed && xmax <= kPairHigh;
  float top = xmax, unused = xmax;
  db_two(top, unused, lv);
  if (top_db > 0.0f) lv.thr = (isnan(top) ? -INFINITY : top) - top_db;
  return lv;
}

// 4 values in, 4 out; the tail and unaligned buffers one by one.
struct Quad {
  float v[4];
};
__device__ __forceinline__ Quad load_quad(const float *x, long long i, long long n, bool vec, float fill) {
  Quad q;
  if (vec && i + 4 <= n) {
    const float4 f = *reinterpret_cast<const float4 *>(x + i);
    q.v[0] = f.x;
    q.v[1] = f.y;
    q.v[2] = f.z;
    q.v[3] = f.w;
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) q.v[k] = i + k < n ? x[i + k] : fill;
  }
  return q;
}
__device__ __forceinline__ void store_quad(float *y, long long i, long long n, bool vec, const Quad &q) {
  if (vec && i + 4 <= n) {
    *reinterpret_cast<float4 *>(y + i) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (i + k < n) y[i + k] = q.v[k];
  }
}
// dB values of a quad with their floor.
__device__ __forceinline__ void db_quad(Quad &q, const Levels &lv, bool floor_on) {
  db_two(q.v[0], q.v[1], lv);
  db_two(q.v[2], q.v[3], lv);
  if (floor_on) {
#pragma unroll
    for (int k = 0; k < 4; k++) q.v[k] = vthr(q.v[k], lv.thr);
  }
}
__device__ __forceinline__ bool aligned16(const void *p) { return (reinterpret_cast<size_t>(p) & 15) == 0; }

// x and y may be the same buffer: a thread reads what it writes, before it.
__global__ void __launch_bounds__(kDbSmallThreads) db_small_kernel(const float *x, float *y, long long n, float mult,
                                                                   float amin, float ref, bool ref_max, float top_db) {
  const bool vx = aligned16(x), vy = aligned16(y);
  Quad q[kDbSmallPer];
  float vmax = -INFINITY;
  bool nan = false;
#pragma unroll
  for (int u = 0; u < kDbSmallPer; u++) {
    q[u] = load_quad(x, 4LL * (threadIdx.x + u * kDbSmallThreads), n, vx, -INFINITY);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      vmax = fmaxf(vmax, q[u].v[k]);
      nan |= isnan(q[u].v[k]);
    }
  }
  block_max<kDbSmallThreads>(vmax, nan);
  const Levels lv = levels_of_max(vmax, nan, ref, ref_max, mult, amin, top_db);
#pragma unroll
  for (int u = 0; u < kDbSmallPer; u++) {
    const long long i = 4LL * (threadIdx.x + u * kDbSmallThreads);
    if (i >= n) break;
    db_quad(q[u], lv, top_db > 0.0f);
    store_quad(y, i, n, vy, q[u]);
  }
}

// part[b] = {max of block b's share of x (NaNs skipped), 1 if it holds a NaN}
__global__ void __launch_bounds__(kDbThreads) db_max_kernel(const float *x, long long n, float2 *part) {
  const bool vx = aligned16(x);
  float vmax = -INFINITY;
  bool nan = false;
  const long long step = 4LL * kDbThreads * gridDim.x;
  long long i = 4LL * (blockIdx.x * (long long)kDbThreads + threadIdx.x);
  for (; i + 3 * step < n; i += 4 * step) {  // four loads in flight
    Quad q[4];
#pragma unroll
    for (int u = 0; u < 4; u++) q[u] = load_quad(x, i + u * step, n, vx, -INFINITY);
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        vmax = fmaxf(vmax, q[u].v[k]);
        nan |= isnan(q[u].v[k]);
      }
  }
  for (; i < n; i += step) {
    const Quad q = load_quad(x, i, n, vx, -INFINITY);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      vmax = fmaxf(vmax, q.v[k]);
      nan |= isnan(q.v[k]);
    }
  }
  block_max<kDbThreads>(vmax, nan);
  if (threadIdx.x == 0) part[blockIdx.x] = make_float2(vmax, nan ? 1.0f : 0.0f);
}

// n_part == 0: no maximum is needed (ref given, no floor).
__global__ void __launch_bounds__(kDbThreads) db_apply_kernel(const float *x, float *y, long long n, float mult,
                                                              float amin, float ref, bool ref_max, float top_db,
                                                              const float2 *part, int n_part) {
  Levels lv = levels(mult, amin, ref);
  if (n_part > 0) {
    float vmax = -INFINITY;
    bool nan = false;
    for (int b = threadIdx.x; b < n_part; b += kDbThreads) {
      const float2 p = __ldg(part + b);
      vmax = fmaxf(vmax, p.x);
      nan |= p.y != 0.0f;
    }
    block_max<kDbThreads>(vmax, nan);
    lv = levels_of_max(vmax, nan, ref, ref_max, mult, amin, top_db);
  }
  const bool floor_on = top_db > 0.0f, vx = aligned16(x), vy = aligned16(y);
  const long long quads = (n + 3) / 4, step = (long long)kDbThreads * gridDim.x;
  // from the end, which db_max_kernel read last; two loads in flight
  long long j = blockIdx.x * (long long)kDbThreads + threadIdx.x;
  for (; j + step < quads; j += 2 * step) {
    const long long i = 4 * (quads - 1 - j), i2 = i - 4 * step;
    Quad q = load_quad(x, i, n, vx, 0.0f), q2 = load_quad(x, i2, n, vx, 0.0f);
    db_quad(q, lv, floor_on);
    store_quad(y, i, n, vy, q);
    db_quad(q2, lv, floor_on);
    store_quad(y, i2, n, vy, q2);
  }
  if (j < quads) {
    const long long i = 4 * (quads - 1 - j);
    Quad q = load_quad(x, i, n, vx, 0.0f);
    db_quad(q, lv, floor_on);
    store_quad(y, i, n, vy, q);
  }
}

// ---- pass by pass (amin <= 0): reference, log + running maximum, floor
// ref_slot (optional): {encoded max of x, NaN flag} written by db_ref_kernel;
// the reference value is then max(x) (NaN when x holds one), as ref=np.max.
__global__ void __launch_bounds__(kDbThreads) db_pass1_kernel(const float *x, float *y, long long n, float mult,
                                                              float amin, float ref, const unsigned *ref_slot,
                                                              unsigned *slot) {
  if (ref_slot) ref = ref_slot[1] ? __int_as_float(0x7fc00000) : dec_f(ref_slot[0]);
  float vmax = -INFINITY;
  for (long long i = blockIdx.x * (long long)kDbThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kDbThreads) {
    const float v = db_value(x[i], mult, amin, ref);
    y[i] = v;
    vmax = fmaxf(vmax, v);
  }
  bool none = false;
  block_max<kDbThreads>(vmax, none);
  if (threadIdx.x == 0 && vmax > -INFINITY) atomicMax(slot, enc_f(vmax));
}

__global__ void __launch_bounds__(kDbThreads) db_ref_kernel(const float *x, long long n, unsigned *ref_slot) {
  float vmax = -INFINITY;
  bool nan = false;
  for (long long i = blockIdx.x * (long long)kDbThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kDbThreads) {
    nan |= isnan(x[i]);
    vmax = fmaxf(vmax, x[i]);
  }
  block_max<kDbThreads>(vmax, nan);
  if (threadIdx.x == 0) {
    if (nan) atomicOr(ref_slot + 1, 1u);
    atomicMax(ref_slot, enc_f(vmax));
  }
}

__global__ void __launch_bounds__(kDbThreads) db_pass2_kernel(float *y, long long n, float top_db,
                                                              const unsigned *slot) {
  const float thr = dec_f(*slot) - top_db;
  for (long long i = blockIdx.x * (long long)kDbThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kDbThreads)
    y[i] = vthr(y[i], thr);
}

__global__ void db_slots_kernel(unsigned *slots, unsigned lowest) {
  slots[0] = slots[1] = lowest;
  slots[2] = 0u;
}

cudaError_t launch_passes(const float *x, float *y, long long n, float mult, float amin, float ref, bool ref_max,
                          float top_db, unsigned *slots, unsigned grid, cudaStream_t s) {
  db_slots_kernel<<<1, 1, 0, s>>>(slots, encode_max_init());
  if (ref_max) db_ref_kernel<<<grid, kDbThreads, 0, s>>>(x, n, slots + 1);
  db_pass1_kernel<<<grid, kDbThreads, 0, s>>>(x, y, n, mult, amin, ref, ref_max ? slots + 1 : nullptr, slots);
  if (top_db > 0.0f) db_pass2_kernel<<<grid, kDbThreads, 0, s>>>(y, n, top_db, slots);
  return cudaGetLastError();
}

constexpr int kDbBlocks = 148 * 8;

}  // namespace

// Whether the maximum of x has to be known, and whether one CTA does it all.
static bool db_needs_max(bool ref_max, float top_db) { return ref_max || top_db > 0.0f; }

size_t db_scratch_bytes(long long n, float amin, bool ref_max, float top_db) {
  if (!(amin > 0.0f)) return 4 * sizeof(unsigned);
  if (n <= kDbSmallMax || !db_needs_max(ref_max, top_db)) return 0;
  return kDbBlocks * sizeof(float2);
}

cudaError_t launch_db(const float *x, float *y, long long n, float mult, float amin, float ref, bool ref_max,
                      float top_db, void *scratch, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (!(amin > 0.0f)) {
    const long long g = (n + kDbThreads - 1) / kDbThreads;
    return launch_passes(x, y, n, mult, amin, ref, ref_max, top_db, static_cast<unsigned *>(scratch),
                         (unsigned)(g < 148 * 16 ? g : 148 * 16), s);
  }
  if (n <= kDbSmallMax) {
    db_small_kernel<<<1, kDbSmallThreads, 0, s>>>(x, y, n, mult, amin, ref, ref_max, top_db);
    return cudaGetLastError();
  }
  const long long quads = (n + 3) / 4, g = (quads + kDbThreads - 1) / kDbThreads;
  const int grid = (int)(g < kDbBlocks ? g : kDbBlocks);
  float2 *part = static_cast<float2 *>(scratch);
  const bool need = db_needs_max(ref_max, top_db);
  if (need) db_max_kernel<<<grid, kDbThreads, 0, s>>>(x, n, part);
  db_apply_kernel<<<grid, kDbThreads, 0, s>>>(x, y, n, mult, amin, ref, ref_max, top_db, part, need ? grid : 0);
  return cudaGetLastError();
}

}  // namespace mm
