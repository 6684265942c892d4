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
// Bound by HBM: 42.3 M values (169 MB, more than L2) with ref = max(x): see the
// figures at launch_db.
//
// amin <= 0 (or NaN) keeps the pass-by-pass form: a logarithm of a negative
// number is NaN and the maximum must skip it.
#include <math.h>

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

// Reference value and floor from max(x) (NaNs skipped) and "x holds a NaN".
__device__ __forceinline__ void db_levels(float xmax, bool nan, bool ref_max, float mult, float amin, float top_db,
                                          float &ref, float &thr) {
  if (ref_max) ref = nan ? __int_as_float(0x7fc00000) : xmax;
  const float top = db_value(xmax, mult, amin, ref);
  thr = top_db > 0.0f ? (isnan(top) ? -INFINITY : top) - top_db : -INFINITY;
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
  float thr;
  db_levels(vmax, nan, ref_max, mult, amin, top_db, ref, thr);
  const bool floor_on = top_db > 0.0f;
#pragma unroll
  for (int u = 0; u < kDbSmallPer; u++) {
    const long long i = 4LL * (threadIdx.x + u * kDbSmallThreads);
    if (i >= n) break;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float v = db_value(q[u].v[k], mult, amin, ref);
      q[u].v[k] = floor_on ? vthr(v, thr) : v;
    }
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
  float thr = -INFINITY;
  if (n_part > 0) {
    float vmax = -INFINITY;
    bool nan = false;
    for (int b = threadIdx.x; b < n_part; b += kDbThreads) {
      const float2 p = __ldg(part + b);
      vmax = fmaxf(vmax, p.x);
      nan |= p.y != 0.0f;
    }
    block_max<kDbThreads>(vmax, nan);
    db_levels(vmax, nan, ref_max, mult, amin, top_db, ref, thr);
  }
  const bool floor_on = top_db > 0.0f, vx = aligned16(x), vy = aligned16(y);
  const long long quads = (n + 3) / 4, step = (long long)kDbThreads * gridDim.x;
  for (long long j = blockIdx.x * (long long)kDbThreads + threadIdx.x; j < quads; j += step) {
    const long long i = 4 * (quads - 1 - j);  // from the end: what db_max_kernel read last
    Quad q = load_quad(x, i, n, vx, 0.0f);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float v = db_value(q.v[k], mult, amin, ref);
      q.v[k] = floor_on ? vthr(v, thr) : v;
    }
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
