// Frame-pair front-end kernels (launch variant 3, n_fft 256..4096, MFCC path):
// framing + periodic Hann + real FFT + |X|^2 + Slaney mel + log10, two
// consecutive frames per group of lanes, with a running per-clip maximum for
// top_db.
//
// The reference computes the same per frame on the CPU, one frame after the
// other (STFT.swift:287-335 window/FFT/power, MelSpectrogram.swift:122-138 mel,
// Scaling.swift:73-118 dB).  Here TPF = n_fft/64 lanes own frames t and t + 1;
// each lane holds 32 complex points of both packed sequences
// z[n] = x[2n] w[2n] + i x[2n+1] w[2n+1] (M = n_fft/2 points), frame t in lane
// 0 and frame t + 1 in lane 1 of packed float32 registers:
//
//   n = j + TPF r   (j = lane in the frame group, r = register)
//   k = k1 + 32 k2
//   stage 1: 32-point DFT over r in registers       -> Y[j][k1]
//            twiddle W_M^(j k1)
//   one shared-memory transpose of 16-byte elements (re, im of both frames),
//   rows of 33 (conflict-free)
//   stage 2: TPF-point DFTs over j in registers      -> Z[k1 + 32 k2]
//   real split X[k] = E + W_N^k O, X[M-k] = conj(E - W_N^k O), both from the
//   pair (Z[k], Z[M-k]): the stage-2 columns are dealt to lanes so that k1
//   and 32-k1 sit in the same lane (TPF < 32); for TPF = 32 the partner lanes
//   l and 32-l swap the upper 16 registers by shuffle and each takes 16 pairs.
// n_fft 4096 has 64 lanes, a warp pair (frame_pair4096_kernel below).
//
// Only warp-level (4096: warp-pair) synchronisation is used.  The window is staged in shared
// memory halved (exact in binary floating point), so the real split's
// E + W O, formed without its factor 1/2, is X itself and the spectrum is
// |X|^2, bit for bit the values of the unscaled transform divided by 4: a bin
// overflows float32 only where the reference's |X|^2 does.
//
// Why two frames.  The single-frame form of this kernel (one frame per warp at
// n_fft 2048, 16 warps an SM) was held by the shared-memory pipe (82 % of its
// wavefronts) and by issue (68 %).  A pair reads the window, twiddles and
// filterbank weights once for two frames, its samples overlap in registers
// (hop n_fft/4: 40 loads a lane instead of 64) and packed arithmetic halves
// the issue slots: 2 075 -> 1 200 warp instructions and ~610 -> 480
// shared-memory wavefronts a frame.  The price is the register file: 128
// registers of data a lane leave 8 warps an SM, and with two warps a scheduler
// the kernel now waits on its own latencies (issue 45 %, L1 / shared-memory
// pipe 74 %).  256 clips of 30 s at n_fft 2048, hop 512, 128 bands: 0.90 -> 0.76
// ms (whole step 0.954 -> 0.81); 512 clips of 10 s at n_fft 512, hop 160, 80
// bands, whole step: 0.62 (CTA-tile kernel) -> 0.39.  64 clips of 30 s at 44.1 kHz,
// n_fft 4096, hop 1024: 0.571 -> 0.511 (one frame per warp pair, 16 warps, before).
// Measured and left out (128 clips, whole step, against 0.426 ms): 12 warps of
// 168 registers 0.443; the next pair's samples loaded into registers before
// the walk 0.445 against 0.438; the next pair's 16-point DFTs interleaved with
// the walk 0.52 (spills and register moves).
#include <math.h>

#include <atomic>

#include "async_copy.cuh"
#include "f32x2.cuh"
#include "frame_common.cuh"
#include "kernels.h"
#include "warp_common.cuh"

namespace mm {

// Float pairs per 32 bins of a pair's spectrum: 34, so that a lane's bins are
// 16-byte aligned; 33 for a warp pair, whose store pattern needs it odd.
__host__ __device__ constexpr int pair_ps(int tpf) { return tpf == 64 ? 33 : 34; }
constexpr float k10Log10of2 = 3.0102999566398120f;  // 10 log10(2)

template <int LOG2N>
struct PShape {
  static constexpr int N = 1 << LOG2N;
  static constexpr int M = N / 2;
  static constexpr int TPF = M / 32;    // lanes per frame pair
  static constexpr int FPW = 32 / TPF;  // frame pairs per warp
  static constexpr int C = FPW;         // stage-2 columns per lane
  static constexpr int HALF = C / 2;
  static constexpr int NW = 8;          // warps per CTA at most, one CTA per SM
  static constexpr int UF = 2 * FPW;     // frames of a warp's unit of work
  static constexpr int UT = 4;           // units per tile of the batch's tile table
  static constexpr int F = UF * UT;      // frames per tile
  static constexpr int MEL_SMEM_MAX = 1024;  // band or packed-weight words staged in shared memory up to this
  // 16-byte slots of a pair's buffer: TPF rows of 33 (at TPF 8 with room for
  // the groups' offsets of P, below); at TPF 32 rows of 32 with the columns
  // of row j swapped within groups of 8 by XOR with j mod 8 (both ways of
  // access conflict-free)
  static constexpr int BS = TPF == 32 ? 1024 : TPF * 33 + (TPF == 8 ? 16 : 0);
  static constexpr int PS = pair_ps(TPF);
  static_assert(TPF >= 4 && TPF <= 32, "n_fft must be 256..2048");
};

// Real-split factors of lane l (one pair per warp only), see below: 512 x 2
// floats, staged as float4 of i = 2p, 2p + 1 at [32 p + l].
template <int LOG2N>
__host__ __device__ constexpr size_t pair_split_tw() {
  return PShape<LOG2N>::C == 1 ? size_t(16 * 32) * 8 : 0;
}

template <int LOG2N>
__host__ __device__ constexpr size_t pair_fixed_smem() {
  using S = PShape<LOG2N>;
  return size_t(16) * S::TPF * 16 + align16(size_t(S::N) * 4) + pair_split_tw<LOG2N>();
}
// ... and per warp
template <int LOG2N>
__host__ __device__ constexpr size_t pair_warp_smem() {
  return size_t(PShape<LOG2N>::FPW) * PShape<LOG2N>::BS * 16;
}

// n_fft 4096: a pair of frames on a warp pair (frame_pair4096_kernel)
struct P4Shape {
  static constexpr int N = 4096, M = N / 2, TPF = 64;
  static constexpr int NP = 4;  // warp pairs per CTA, one CTA per SM
  static constexpr int UF = 2, UT = 4;
  static constexpr int BS = TPF * 33;  // 16-byte slots of a buffer
  static constexpr int PS = pair_ps(TPF);
  static constexpr int RS = 16 * 33;   // real-split factors, rows of 33
  static constexpr int MEL_SMEM_MAX = 1024;
  static constexpr size_t fixed = size_t(16) * TPF * 16 + size_t(N) * 4 + size_t(RS) * 16;
  static constexpr size_t walk = (16 * 24 + 16) * size_t(TPF);
  static_assert(PS * TPF * 8 % 16 == 0 && PS * TPF / 2 + 1024 <= BS, "spectrum and 1 024 parts fit the buffer");
};

int warp_frames_per_tile(int log2n) {
  switch (log2n) {
    case 8: return PShape<8>::F;
    case 9: return PShape<9>::F;
    case 10: return PShape<10>::F;
    case 11: return PShape<11>::F;
    case 12: return P4Shape::UF * P4Shape::UT;
    default: return 0;
  }
}

// Samples (x[i], x[i+1]) for i = first + stride r, r < Q, with the padding
// rule; used only for frames that overlap the clip's edges.  Out of line, so
// that its index arithmetic does not weigh on the interior path, and fully
// unrolled, so that its loads are in flight together (a short clip waits for
// its edges).
template <int Q>
__device__ __noinline__ void gather_edge_n(float2 *out, const float *sig, long long first, long long L, int pad_mode,
                                           int stride) {
  const long long last = first + (long long)stride * (Q - 1) + 1;
  // the clip as offsets [lo, hi) from `first` (the offsets asked for are small)
  constexpr long long kFar = 1 << 30;
  const int lo = (int)max(min(-first, kFar), -kFar), hi = (int)max(min(L - first, kFar), -kFar);
  const float *p = sig + first;
  if (pad_mode != PAD_REFLECT) {
#pragma unroll
    for (int r = 0; r < Q; r++) {
      const int i = stride * r;
      float x = 0.0f, y = 0.0f;
      if (i >= lo && i < hi) x = __ldg(p + i);
      if (i + 1 >= lo && i + 1 < hi) y = __ldg(p + i + 1);
      out[r] = make_float2(x, y);
    }
  } else if (first > -L && last <= 2 * (L - 1)) {  // one reflection at most
    auto at = [&](int i) { return i < lo ? 2 * lo - i : (i >= hi ? 2 * (hi - 1) - i : i); };
#pragma unroll
    for (int r = 0; r < Q; r++) out[r] = make_float2(__ldg(p + at(stride * r)), __ldg(p + at(stride * r + 1)));
  } else {  // a clip shorter than the padding
    for (int r = 0; r < Q; r++) {
      const long long n0 = first + (long long)stride * r;
      out[r] = make_float2(sample_at(sig, n0, L, pad_mode), sample_at(sig, n0 + 1, L, pad_mode));
    }
  }
}

// The filterbank walk's sums (R, F) into a part slot.  (No memory clobber:
// the slots lie outside the spectrum, whose loads may then be issued ahead of
// the stores; a warp barrier stands before the slots are read.)
__device__ __forceinline__ void walk_store(uint32_t at, f2 R, f2 F) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(at), "l"(R.v), "l"(F.v));
}
// Where bit G of fl is set: the sums into slot `at`, and new ones from bin p.
template <int G>
__device__ __forceinline__ void walk_end(f2 p, float wr, float wf, unsigned fl, f2 &R, f2 &F, uint32_t &at) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t.reg .b32 t;\n\t"
      "and.b32 t, %3, %4;\n\t"
      "setp.ne.u32 q, t, 0;\n\t"
      "@q st.shared.v2.b64 [%2], {%0, %1};\n\t"
      "@q add.u32 %2, %2, 16;\n\t"
      "@q mul.rn.f32x2 %0, %5, %6;\n\t"
      "@q mul.rn.f32x2 %1, %5, %7;\n\t}"
      : "+l"(R.v), "+l"(F.v), "+r"(at)
      : "r"(fl), "n"((int)(1u << G)), "l"(p.v), "l"(dup2(wr).v), "l"(dup2(wf).v));
}

// Position of bin k in a pair's padded spectrum.
template <int TPF>
__device__ __forceinline__ int pair_bin(int k) {
  const int q = k >> 5;
  return k + (pair_ps(TPF) - 32) * (q < TPF - 1 ? q : TPF - 1);
}

// Synchronisation of the lanes that own a pair: part of a warp (any() of the
// lanes in `mask`), or the 64 threads of a warp pair on named barrier id + 1.
struct GroupSync {
  unsigned mask;
  __device__ __forceinline__ void operator()() const { __syncwarp(); }
  __device__ __forceinline__ bool any(bool p) const { return (__ballot_sync(0xffffffffu, p) & mask) != 0; }
};
struct WarpPairSync {
  int id;
  __device__ __forceinline__ void operator()() const { frame_sync<64>(id); }
  __device__ __forceinline__ bool any(bool p) const { return frame_sync_or<64>(id, p); }
};

// Tables of the filterbank walk (walk_bands) in shared memory.
struct WalkTables {
  const float4 *wa;   // [16][TPF]
  const float2 *wb;   // [16][TPF]
  const int4 *lane;   // [TPF]
  const int *band;
  bool twice;         // some pair of bins ends two segments
};

// Stages them from the lane tables (build_mel_lane_kernel), lane-minor: per
// pair of bins g < 16 of lane l the weights (rising, falling) of the first bin
// and of the second in the segment that is open (wa), and of the second in a
// segment it starts (wb); and the lane words.  True when this thread saw a
// pair of bins that ends two segments.
template <int TPF>
__device__ __forceinline__ bool stage_walk(const FrontArgs &a, float4 *wa, float2 *wb, int4 *lane_s, int tid,
                                           int threads) {
  bool twice = false;
  // flush bits of a lane's bins, bin 31 left to the end of the walk
  auto flush_bit = [&](int2 w, int bin) { return bin < 31 ? ((unsigned)w.x >> bin) & 1u : 0u; };
  for (int i = tid; i < TPF; i += threads) {
    const int2 w = __ldg(a.mel_lane + i);
    unsigned m1 = 0u, m2 = 0u;
    for (int g = 0; g < 16; g++) {
      const unsigned fa = flush_bit(w, 2 * g), fb = flush_bit(w, 2 * g + 1);
      m1 |= (fa | fb) << g;
      m2 |= (fa & fb) << g;
    }
    // {first | second segment end by pair, first part's byte offset, parts the
    // head takes over from the next lanes, the empty segments' slot}
    lane_s[i] = make_int4((int)(m1 | m2 << 16), 16 * (w.y & 1023), (w.y >> 10) & 63, w.y >> 16);
    if (m2) twice = true;
  }
  for (int i = tid; i < 16 * TPF; i += threads) {
    const int g = i / TPF, j = i - g * TPF;
    const bool fa = flush_bit(__ldg(a.mel_lane + j), 2 * g) != 0;
    const float2 u = __ldg(a.mel_lw + 2 * g * TPF + j), w = __ldg(a.mel_lw + (2 * g + 1) * TPF + j);
    wa[i] = make_float4(u.x, u.y, fa ? 0.0f : w.x, fa ? 0.0f : w.y);
    wb[i] = make_float2(fa ? w.x : 0.0f, fa ? w.y : 0.0f);
  }
  return twice;
}

// A band's dB value of both frames into their rows, and the running maximum.
__device__ __forceinline__ void put_band(const FrontArgs &a, f2 sum, int m, float ref_db, float *dst, bool va, bool vb,
                                         float &vmax) {
  float xa, xb;
  un2(sum, xa, xb);
  const float da = fmaf(k10Log10of2, __log2f(fmaxf(xa, a.amin)), -ref_db);
  const float db = fmaf(k10Log10of2, __log2f(fmaxf(xb, a.amin)), -ref_db);
  if (va) {
    dst[m] = da;
    vmax = fmaxf(vmax, da);
  }
  if (vb) {
    dst[a.n_mels + m] = db;
    vmax = fmaxf(vmax, db);
  }
}

// The filterbank walk.  Lane l sums its 32 bins (the last lane also the
// Nyquist bin) into (R, F) = (rising, falling weight) times P and stores the
// sums in the next part slot at every segment end.  Bins go in pairs: the
// second bin of a pair has its weights in one of two sets, zero in the other,
// wa.zw for the segment that the first bin belongs to and wb for a segment
// that it starts, so one predicated store and restart serve a pair wherever in
// it the segment ends.  Pairs that end two segments (bands of a single bin)
// take the second end in a branch of their own.
template <int TPF, typename Sync>
__device__ __forceinline__ void walk_bands(const FrontArgs &a, const Sync &sync, const f2 *P, cpx2 *parts, int l,
                                           const WalkTables &w, float ref_db, float *dst, bool va, bool vb,
                                           float &vmax) {
  const int4 li = w.lane[l];
  const unsigned fl = (unsigned)li.x;
  const uint32_t part0 = smem_u32(parts);
  uint32_t at = part0 + (unsigned)li.y;  // the next part's slot
  const f2 *pl = P + pair_ps(TPF) * l;
  auto bins = [&](int g) {  // bins 2g, 2g + 1 of both frames
    if constexpr (pair_ps(TPF) % 2 == 0) return reinterpret_cast<const float4 *>(pl)[g];
    else return make_float4(lo2(pl[2 * g]), hi2(pl[2 * g]), lo2(pl[2 * g + 1]), hi2(pl[2 * g + 1]));
  };
  const float4 *wa = w.wa + l;
  const float2 *wb = w.wb + l;
  const f2 zero = dup2(0.0f);
  f2 R = zero, Fs = zero;
  // the frames' non-finite check: the largest bit pattern of a power (a power
  // is never negative; NaN and inf lie at or above inf's pattern)
  unsigned mxa = 0u, mxb = 0u;
  static_for<0, 16>([&](auto gi) {
    constexpr int g = decltype(gi)::value;
    const float4 pq = bins(g), u = wa[g * TPF];
    const float2 v = wb[g * TPF];
    mxa = max(max(mxa, __float_as_uint(pq.x)), __float_as_uint(pq.z));
    mxb = max(max(mxb, __float_as_uint(pq.y)), __float_as_uint(pq.w));
    const f2 p0 = pk2(pq.x, pq.y), p1 = pk2(pq.z, pq.w);
    R = fma2(p0, dup2(u.x), R);
    Fs = fma2(p0, dup2(u.y), Fs);
    R = fma2(p1, dup2(u.z), R);
    Fs = fma2(p1, dup2(u.w), Fs);
    walk_end<g>(p1, v.x, v.y, fl, R, Fs, at);
    if (w.twice && (fl & (0x10000u << g))) {
      walk_store(at, R, Fs);
      at += 16;
      R = zero;
      Fs = zero;
    }
  });
  if (l == TPF - 1) {
    if (__ldg(a.mel_lane + l).x < 0) {  // bin 31 ends a segment
      walk_store(at, R, Fs);
      at += 16;
      R = zero;
      Fs = zero;
    }
    float pa, pb2;
    un2(pl[32], pa, pb2);
    const float2 wn = __ldg(a.mel_lw + 32 * TPF + l);
    mxa = max(mxa, __float_as_uint(pa));
    mxb = max(mxb, __float_as_uint(pb2));
    R = fma2(pl[32], dup2(wn.x), R);
    Fs = fma2(pl[32], dup2(wn.y), Fs);
  }
  walk_store(at, R, Fs);
  if (l == 0) parts[li.w] = {zero, zero};  // the empty segments' slot
  const bool bada = sync.any(mxa >= 0x7f800000u), badb = sync.any(mxb >= 0x7f800000u);
  // added to a frame's band sums: NaN where a bin of it is not finite
  const float qnan = __int_as_float(0x7fc00000);
  const f2 nan2 = pk2(bada ? qnan : 0.0f, badb ? qnan : 0.0f);
  sync();
  // a lane whose last part heads a segment adds the parts of the lanes the
  // segment runs into
  if (li.z) {
    cpx2 *h = parts + ((at - part0) >> 4);
    cpx2 hv = *h;
    for (int j = 1; j <= li.z; j++) hv = cadd(hv, h[j]);
    *h = hv;
  }
  sync();
  // band m is the head of segment m (rising) plus the head of segment m + 1
  // (falling); four bands at a time, so that their reads overlap.  The lane
  // tables hold finite weights only: no band is NaN by itself.
  const char *pb = reinterpret_cast<const char *>(parts);
  for (int m0 = l; m0 < a.n_mels; m0 += 4 * TPF) {
    int bw[4];
    f2 acc[4];
#pragma unroll
    for (int i = 0; i < 4; i++) bw[i] = m0 + i * TPF < a.n_mels ? w.band[m0 + i * TPF] : 0;
#pragma unroll
    for (int i = 0; i < 4; i++)
      acc[i] = add2(*reinterpret_cast<const f2 *>(pb + 16 * (bw[i] & 4095)),
                    *reinterpret_cast<const f2 *>(pb + 8 + 16 * ((bw[i] >> 12) & 4095)));
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int m = m0 + i * TPF;
      put_band(a, add2(acc[i], nan2), m, ref_db, dst, va && m < a.n_mels, vb && m < a.n_mels, vmax);
    }
  }
}

// The bands of a filterbank that the lane tables cannot describe, from packed rows.
template <int TPF, typename Sync>
__device__ __forceinline__ void row_bands(const FrontArgs &a, const Sync &sync, const f2 *P, int l, const float *melw,
                                          float ref_db, float *dst, bool va, bool vb, float &vmax) {
  unsigned mxa = 0u, mxb = 0u;  // the non-finite check: this lane's share of the bins
  for (int k = l; k <= 32 * TPF; k += TPF) {
    float pa, pb;
    un2(P[pair_bin<TPF>(k)], pa, pb);
    mxa = max(mxa, __float_as_uint(pa));
    mxb = max(mxb, __float_as_uint(pb));
  }
  const bool bada = sync.any(mxa >= 0x7f800000u), badb = sync.any(mxb >= 0x7f800000u);
  const float qnan = __int_as_float(0x7fc00000);
  for (int m = l; m < a.n_mels; m += TPF) {
    const int4 info = __ldg(a.mel_info + m);
    const float *wr = melw + info.z;
    f2 acc = dup2(0.0f);
    for (int q = 0; q < info.y; q++) acc = fma2(P[pair_bin<TPF>(info.x + q)], dup2(wr[q]), acc);
    acc = add2(acc, pk2(info.w || bada ? qnan : 0.0f, info.w || badb ? qnan : 0.0f));
    put_band(a, acc, m, ref_db, dst, va, vb, vmax);
  }
}

// Samples (x[2n], x[2n+1]), n = l + TPF r, r < n_q, of the frame that starts at
// s0 (and, with the overlap of the next, `reach` samples more).
template <int TPF, bool EVEN, int NQ>
__device__ __forceinline__ void gather_frame(float2 (&q)[NQ], const FrontArgs &a, const ClipDesc &cd, long long s0,
                                             int reach, int l) {
  const float *base = a.signal + cd.sig_off + s0 + 2 * l;
  if (s0 >= 0 && s0 + reach + 64 * TPF <= cd.length) {
    if (EVEN || ((cd.sig_off + s0) & 1) == 0) {
#pragma unroll
      for (int r = 0; r < NQ; r++) q[r] = __ldg(reinterpret_cast<const float2 *>(base + 2 * TPF * r));
    } else {
#pragma unroll
      for (int r = 0; r < NQ; r++) q[r] = make_float2(__ldg(base + 2 * TPF * r), __ldg(base + 2 * TPF * r + 1));
    }
  } else {  // frames that reach into the padding (a few per clip)
    float2 te[NQ];
    gather_edge_n<NQ>(te, a.signal + cd.sig_off, s0 + 2 * l, cd.length, a.pad_mode, 2 * TPF);
#pragma unroll
    for (int r = 0; r < NQ; r++) q[r] = te[r];
  }
}

// Both frames times the window; even registers into e, odd ones into o.
template <int TPF>
__device__ __forceinline__ void window_pair(const float2 *qa, const float2 *qb, const float4 *wl, cpx2 *e, cpx2 *o) {
#pragma unroll
  for (int r = 0; r < 32; r += 2) {
    const float4 w = wl[TPF * (r / 2)];
    e[r / 2] = {pk2(qa[r].x * w.x, qb[r].x * w.x), pk2(qa[r].y * w.y, qb[r].y * w.y)};
    o[r / 2] = {pk2(qa[r + 1].x * w.z, qb[r + 1].x * w.z), pk2(qa[r + 1].y * w.w, qb[r + 1].y * w.w)};
  }
}

// Frames t and t + 1 gathered and windowed (D: see frame_pair_kernel).
template <int TPF, int D>
__device__ __forceinline__ void load_pair(const FrontArgs &a, const ClipDesc &cd, int t, int l, const float4 *win_s,
                                          cpx2 *e, cpx2 *o) {
  const long long s0 = (long long)t * a.hop - a.pad;
  float2 q[D > 0 ? 32 + D : 32];
  gather_frame<TPF, (D > 0)>(q, a, cd, s0, D > 0 ? a.hop : 0, l);
  if constexpr (D > 0) {
    window_pair<TPF>(q, q + D, win_s + l, e, o);
  } else {
    float2 qb[32];
    gather_frame<TPF, false>(qb, a, cd, s0 + a.hop, 0, l);
    window_pair<TPF>(q, qb, win_s + l, e, o);
  }
}

// The last butterflies of a pair's stage 1 (e, o: its two 16-point DFTs), each
// followed by the twiddle W_M^(j k1) of row j (tw at [k TPF]) and put(k1, value).
template <int TPF, typename Put>
__device__ __forceinline__ void finish_stage1(const cpx2 *e, const cpx2 *o, const float4 *tw, Put &&put) {
  static_for<0, 16>([&](auto ki) {
    constexpr int k = decltype(ki)::value;
    using R = Rot<k, 32>;
    cpx2 lo, hi;
    rot_butterfly<R>(e[k], R::rot(o[k]), lo, hi);
    const float4 tk = tw[k * TPF];
    if constexpr (k > 0) lo = cmul(lo, {tk.x, tk.y});
    hi = cmul(hi, {tk.z, tk.w});
    put(std::integral_constant<int, k>{}, lo);
    put(std::integral_constant<int, k + 16>{}, hi);
  });
}

// |X[k]|^2 and |X[M-k]|^2 of both frames from za = Z[k], zb = Z[M-k] and the
// factors (scale, ratio) of W_N^k: (cos, tan) below an eighth of a turn (LOW),
// (sin, cot) above.  The window was halved.
template <bool LOW>
__device__ __forceinline__ void split_pair(cpx2 za, cpx2 zb, float scale, float ratio, f2 &p, f2 &q) {
  const f2 ex = add2(za.x, zb.x), ey = sub2(za.y, zb.y);
  const f2 ox = add2(za.y, zb.y), oy = sub2(zb.x, za.x);
  const f2 sc = dup2(scale), rt = dup2(ratio);
  f2 wr, wi;  // W_N^k O without its scale
  if constexpr (LOW) {
    wr = fma2(oy, rt, ox);
    wi = fma2(neg2(ox), rt, oy);
  } else {
    wr = fma2(ox, rt, oy);
    wi = fma2(oy, rt, neg2(ox));
  }
  const f2 xr = fma2(wr, sc, ex), xi = fma2(wi, sc, ey);
  const f2 yr = fma2(neg2(wr), sc, ex), yi = fma2(neg2(wi), sc, ey);
  p = fma2(xr, xr, mul2(xi, xi));
  q = fma2(yr, yr, mul2(yi, yi));
}

// The factors of split_pair for W_N^k = c - i s as (scale, ratio).
__device__ __forceinline__ float2 split_factors(cpx w, bool low) {
  return low ? make_float2(w.x, -w.y / w.x) : make_float2(-w.y, w.x / -w.y);
}

// The warp's running maximum of clip `clip` into its slot.
__device__ __forceinline__ void flush_max(const FrontArgs &a, int clip, float vmax, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if (lane == 0 && clip >= 0 && vmax > -INFINITY) atomicMax(a.clip_max + clip, enc_f(vmax));
}

// The units of work of one warp (or warp pair): `first`, then every `step`-th
// of this CTA's contiguous range that holds a frame.
template <int UF, int UT>
struct Units {
  int u, end, step;
  int clip = -1, past = -1;  // past: first unit after the current clip
  ClipDesc cd{};
  // A CTA's range is dealt to its warps in turn, so that the samples its warps
  // read at a time overlap.
  __device__ __forceinline__ Units(const FrontArgs &a, int worker, int workers) {
    const long long total = (long long)a.total_tiles * UT;
    u = (int)(blockIdx.x * total / gridDim.x) + worker - workers;
    end = (int)((blockIdx.x + 1) * total / gridDim.x);
    step = workers;
  }
  __device__ __forceinline__ int first_frame() const { return (u - cd.tile_base * UT) * UF; }
  __device__ __forceinline__ bool advance(const FrontArgs &a) {
    while ((u += step) < end) {
      if (u >= past) {  // every frame of a tile belongs to one clip
        clip = __ldg(a.tile_clip + u / UT);
        cd = load_clip(a.clips + clip);
        past = (cd.tile_base + (cd.n_frames + UF * UT - 1) / (UF * UT)) * UT;
      }
      if (first_frame() < cd.n_frames) return true;
    }
    return false;
  }
};

// D > 0: hop = 2 TPF D samples and every clip starts at an even sample, so
// register r of frame t + 1 is register r + D of frame t and the pair's gather
// is 32 + D 8-byte loads a lane; D = 0: any hop and start.
template <int LOG2N, int D>
__global__ void __launch_bounds__(32 * PShape<LOG2N>::NW, 1) frame_pair_kernel(FrontArgs a, int nw) {
  using S = PShape<LOG2N>;
  constexpr int N = S::N, M = S::M, TPF = S::TPF, C = S::C, HALF = S::HALF, PS = S::PS;
  constexpr unsigned FULL = 0xffffffffu;
  griddep_launch();
  extern __shared__ __align__(16) unsigned char smem[];
  const int nmel = a.n_mels;
  const float ref_db = 10.0f * log10f(a.ref);
  // Lane walk over the per-bin split of the filterbank (else packed rows).
  const bool lanes = a.mel_lane_ok != 0;
  constexpr int threads = 32 * S::NW;
  unsigned char *sp = smem;
  // stage-1 twiddles: tw4[k][j] = (W_M^(j k), W_M^(j (k + 16))), k < 16
  float4 *tw4 = reinterpret_cast<float4 *>(sp);
  sp += size_t(16) * TPF * 16;
  // analysis window (halved), the sample pairs of registers r, r + 1 of lane
  // l as one float4 at [r / 2][l]
  float4 *win_s = reinterpret_cast<float4 *>(sp);
  sp += align16(size_t(N) * 4);
  // C == 1: real-split factors (scale, ratio) of W_N^(l + 32 i): cos and tan
  // below an eighth of a turn (i < 8), sin and cot above
  float4 *rs_tw = reinterpret_cast<float4 *>(sp);
  sp += pair_split_tw<LOG2N>();
  // filterbank walk (see there), lane-minor: per pair of bins g < 16 of lane l
  // the weights (rising, falling) of the first bin and of the second in the
  // segment that is open, and of the second in a segment it starts; lane words
  float4 *wa_s = reinterpret_cast<float4 *>(sp);
  if (lanes) sp += size_t(16) * 16 * TPF;
  float2 *wb_s = reinterpret_cast<float2 *>(sp);
  if (lanes) sp += size_t(16) * 8 * TPF;
  int4 *lane_s = reinterpret_cast<int4 *>(sp);
  if (lanes) sp += size_t(16) * TPF;
  cpx2 *bufs = reinterpret_cast<cpx2 *>(sp);
  sp += size_t(nw) * pair_warp_smem<LOG2N>();
  // band words, or the packed rows' weights (their descriptors stay in
  // global memory); past MEL_SMEM_MAX words both stay there
  const int words = lanes ? nmel : a.mel_nnz;
  const bool staged = words <= S::MEL_SMEM_MAX;
  int *words_s = reinterpret_cast<int *>(sp);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = lane / TPF;      // frame pair of this lane within the warp
  const int l = lane - grp * TPF;  // lane within the group
  const float2 *twq = a.tw_split;  // W_N^t, t < N/4

  for (int i = tid; i < 16 * TPF; i += threads) {
    const int k = i / TPF, j = i - k * TPF;
    const cpx u = root_q(twq, 2 * j * k, N), w = root_q(twq, 2 * j * (k + 16), N);
    tw4[i] = make_float4(u.x, u.y, w.x, w.y);
  }
  for (int i = tid; i < 16 * TPF; i += threads) {  // halved: see the header comment
    const int p = i / TPF, j = i - p * TPF;
    const float2 u = __ldg(reinterpret_cast<const float2 *>(a.window) + j + TPF * (2 * p));
    const float2 w = __ldg(reinterpret_cast<const float2 *>(a.window) + j + TPF * (2 * p + 1));
    win_s[i] = make_float4(0.5f * u.x, 0.5f * u.y, 0.5f * w.x, 0.5f * w.y);
  }
  if constexpr (C == 1)
    for (int i = tid; i < 8 * 32; i += threads) {
      const int p = i >> 5, ll = i & 31;
      const cpx u = root_q(twq, ll + 64 * p, N), w = root_q(twq, ll + 32 * (2 * p + 1), N);
      // both entries of p lie on the same side of an eighth of a turn
      const float2 fu = split_factors(u, p < 4), fw = split_factors(w, p < 4);
      rs_tw[i] = make_float4(fu.x, fu.y, fw.x, fw.y);
    }
  bool twice = lanes && stage_walk<TPF>(a, wa_s, wb_s, lane_s, tid, threads);
  const int *src_words = lanes ? a.mel_band : reinterpret_cast<const int *>(a.mel_pw);
  if (staged)
    for (int i = tid; i < words; i += threads) words_s[i] = __ldg(src_words + i);
  const int *band = staged ? words_s : src_words;
  const float *melw = reinterpret_cast<const float *>(band);
  twice = __syncthreads_or(twice) != 0;
  griddep_wait();  // the tables are constant; the clips and their maxima are not
  if (warp >= nw) return;  // a small batch: this warp only helped to stage the tables

  // real-split bases W_N^(first bin of each column pair), C > 1
  cpx base_c[HALF > 0 ? HALF : 1];
  cpx base_hi = {0.0f, 0.0f};
  if constexpr (C > 1) {
#pragma unroll
    for (int c = 0; c < HALF; c++) base_c[c] = root_q(twq, l + TPF * c, N);
    base_hi = (l == 0) ? root_q(twq, 16 + 3 * (N / 4), N) : base_c[0];
  }

  cpx2 *fb = bufs + (warp * S::FPW + grp) * S::BS;
  // both frames' power spectra as float pairs, padded: bin k at
  // k + 2 min(k / 32, TPF - 1), so that lane l reads its bins
  // [32 l, 32 l + 32) as float4 at 17 l + b / 2 and the Nyquist bin is the
  // last lane's 33rd; at TPF 8 the groups start 8 g pairs into their buffers,
  // so that the two groups of a half warp store to disjoint banks
  f2 *P = reinterpret_cast<f2 *>(fb) + (TPF == 8 ? 8 * grp : 0);
  cpx2 *parts = reinterpret_cast<cpx2 *>(P + PS * TPF);  // {R, F} of both frames per part
  const GroupSync sync{(TPF == 32) ? FULL : (((1u << TPF) - 1u) << (grp * TPF))};

  Units<S::UF, S::UT> units(a, warp, nw);  // 2 FPW consecutive frames of one clip each
  int vclip = -1;  // the clip vmax belongs to
  float vmax = -INFINITY;
  while (units.advance(a)) {
    if (units.clip != vclip) {
      flush_max(a, vclip, vmax, lane);
      vclip = units.clip;
      vmax = -INFINITY;
    }
    const ClipDesc &cd = units.cd;
    const int tw0 = units.first_frame(), t = tw0 + 2 * grp;
    const bool va = t < cd.n_frames, vb = t + 1 < cd.n_frames;
    float *dst = a.out + (cd.frame_off + t) * (long long)nmel;

    cpx2 e[16], o[16];
    load_pair<TPF, D>(a, cd, t, l, win_s, e, o);
    // the samples that this warp's next unit adds to the CTA's, into L1: one
    // line a lane (n_fft 1024: 0.459 against 0.466 ms for 128 clips of 30 s)
    {
      const long long o = (long long)(tw0 + S::UF * nw) * a.hop - a.pad + N - (S::UF - 1) * a.hop + lane * 32;
      if (lane * 32 < S::UF * a.hop && o >= 0 && o < cd.length)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.signal + cd.sig_off + o));
    }
    // ---- stage 1: 32-point DFT over registers; its last butterflies are
    // followed directly by the twiddle W_M^(l k1) and the store into row l of
    // the pair's buffer, so that registers free up as it goes.
    dft16(e);
    dft16(o);
    __syncwarp();  // the previous unit's reads of the buffer are done
    {
      cpx2 *row = fb + l * (TPF == 32 ? 32 : 33);
      finish_stage1<TPF>(e, o, tw4 + l, [&](auto ki, cpx2 y) {
        constexpr int k = decltype(ki)::value;
        if constexpr (TPF == 32) row[(k & 24) + ((k & 7) ^ (l & 7))] = y;
        else row[k] = y;
      });
    }
    __syncwarp();
    cpx2 v[32];
    static_for<0, C>([&](auto ci) {
      constexpr int cc = decltype(ci)::value;
      const int col = stage2_col<TPF, C, cc>(l);
#pragma unroll
      for (int jj = 0; jj < TPF; jj++)
        v[cc * TPF + jj] = fb[TPF == 32 ? jj * 32 + (col ^ (jj & 7)) : jj * 33 + col];
    });
    // ---- stage 2: TPF-point DFTs, v[c*TPF + k2] = Z[col(c) + 32 k2]
#pragma unroll
    for (int cc = 0; cc < C; cc++) dft_any<TPF>(v + cc * TPF);
    __syncwarp();  // every lane has read its columns: fb becomes P

    // ---- real split, P[k] = |X[k]|^2 (the window was halved)
    if constexpr (C == 1) {
      // lanes l and 32-l swap registers 16..31: pair i of lane l is
      // (Z[l + 32 i], Z[M - l - 32 i]) = (v[i], partner's v[31 - i]); lane 0
      // pairs with itself: (v[i], v[32 - i]) and the self pair v[16] (k = M/2).
      const int src = (32 - l) & 31;
      const bool l0 = (l == 0);
      f2 *Pa = P + l;  // bin l + 32 i at l + PS i
      // bin M - l - 32 i at M + 2 (TPF - 1) - l - PS i (lane 0, i > 0: 2
      // further on; its i = 0 is the Nyquist bin)
      f2 *Pb = P + (M + 2 * (TPF - 1) - l) + (l0 ? 2 : 0);
      float4 rsp;
      cpx2 prev = v[0];  // lane 0's partner of pair i: its own v[32 - i]
      static_for<0, 16>([&](auto ki) {
        constexpr int i = decltype(ki)::value;
        const cpx2 za = v[i];
        const cpx2 up = v[31 - i];  // sent to the partner; lane 0's own for pair i + 1
        const cpx2 rcv = {shfl2(up.x, src), shfl2(up.y, src)};
        const cpx2 zb = csel(l0, prev, rcv);
        prev = up;
        if constexpr (i % 2 == 0) rsp = rs_tw[32 * (i / 2) + l];
        f2 p, q;
        split_pair<(i < 8)>(za, zb, i % 2 == 0 ? rsp.x : rsp.z, i % 2 == 0 ? rsp.y : rsp.w, p, q);
        Pa[PS * i] = p;
        if constexpr (i == 0) Pb[l0 ? -2 : 0] = q;  // lane 0: the Nyquist bin
        else Pb[-PS * i] = q;
      });
      if (l0) P[M / 2 + TPF] = mul2(dup2(4.0f), fma2(prev.x, prev.x, mul2(prev.y, prev.y)));
    } else {
      const bool l0 = (l == 0);
      static_for<0, HALF>([&](auto ci) {
        constexpr int cc = decltype(ci)::value;
        static_for<0, TPF>([&](auto ki) {
          constexpr int k2 = decltype(ki)::value;
          cpx2 za, zb;
          cpx base;
          int ka;
          if constexpr (cc == 0) {
            constexpr bool lo = k2 < TPF / 2;
            constexpr int ia0 = lo ? k2 : HALF * TPF + (k2 - TPF / 2);
            constexpr int ib0 = lo ? (TPF - k2) % TPF : HALF * TPF + TPF - 1 - (k2 - TPF / 2);
            constexpr int ia = k2, ib = HALF * TPF + TPF - 1 - k2;
            za = csel(l0, v[ia0], v[ia]);
            zb = csel(l0, v[ib0], v[ib]);
            base = lo ? base_c[0] : base_hi;
            ka = l0 ? (lo ? 32 * k2 : 16 + 32 * (k2 - TPF / 2)) : l + 32 * k2;
          } else {
            za = v[cc * TPF + k2];
            zb = v[(cc + HALF) * TPF + TPF - 1 - k2];
            base = base_c[cc];
            ka = l + TPF * cc + 32 * k2;
          }
          const f2 ex = add2(za.x, zb.x), ey = sub2(za.y, zb.y);
          const cpx2 od = {add2(za.y, zb.y), sub2(zb.x, za.x)};
          const cpx2 w = cmul(od, tw_const<k2, 2 * TPF>(base));
          const f2 xr = add2(ex, w.x), xi = add2(ey, w.y);
          const f2 yr = sub2(ex, w.x), yi = sub2(ey, w.y);
          const f2 p = fma2(xr, xr, mul2(xi, xi)), q = fma2(yr, yr, mul2(yi, yi));
          if constexpr (cc == 0) {
            P[l0 ? pair_bin<TPF>(ka) : ka + 2 * k2] = p;
            P[l0 ? pair_bin<TPF>(M - ka) : M - ka + 2 * (TPF - 1 - k2)] = q;
          } else {
            // l + TPF cc + 32 k2 with 0 < l + TPF cc < 32: row k2 and row TPF - 1 - k2
            P[ka + 2 * k2] = p;
            P[M - ka + 2 * (TPF - 1 - k2)] = q;
          }
        });
      });
      if (l0) {
        const cpx2 zm = v[TPF / 2];
        P[M / 2 + TPF] = mul2(dup2(4.0f), fma2(zm.x, zm.x, mul2(zm.y, zm.y)));
      }
    }
    __syncwarp();  // P complete

    // ---- log-mel rows of both frames + running clip max
    if (lanes) walk_bands<TPF>(a, sync, P, parts, l, {wa_s, wb_s, lane_s, band, twice}, ref_db, dst, va, vb, vmax);
    else row_bands<TPF>(a, sync, P, l, melw, ref_db, dst, va, vb, vmax);
  }
  flush_max(a, vclip, vmax, lane);
}

// ---------------------------------------------------------------------------
// n_fft 4096: a pair of frames on a warp pair (64 threads), the same work.
//
//   n = j + 64 r (j < 64: thread of the pair, r < 32), k = k1 + 32 k2 (k2 < 64)
//   stage 1: 32-point DFT over r in registers, twiddle W_M^(j k1), row j of
//            the buffer (16-byte elements, stride 33)
//   stage 2: the 64-point DFT over j of column k1 as 2 x 32: thread (k1, j0)
//            takes rows j0 + 2 j1 (j1 < 32) through a 32-point DFT -> A_j0[q];
//            the two threads of a column (lanes 2i, 2i+1) swap half of their
//            outputs by shuffle, and thread j0 forms
//            Z[k1 + 32 q] = A_0[q] + W_64^q A_1[q] and
//            Z[k1 + 32 (q + 32)] = A_0[q] - W_64^q A_1[q] for q = 2 i + j0.
//   Even columns live in the pair's first warp, odd ones in its second
//   (lane = 2 (k1 >> 1) + j0), so the real-split partner (32 - k1, 1 - j0)
//   of a thread sits in its warp; the two swap their upper 16 registers by
//   shuffle.  Column 0 pairs inside each thread.
// Every shared-memory pattern (row stores, column loads, twiddles, spectrum
// stores, the walk) is conflict-free for this lane assignment.  Bounds as in
// frame_pair_kernel: 8 warps an SM, waiting on their own latencies.
// ---------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(64 * P4Shape::NP, 1) frame_pair4096_kernel(FrontArgs a, int np) {
  using S = P4Shape;
  constexpr int N = S::N, M = S::M, TPF = S::TPF, PS = S::PS, threads = 64 * S::NP;
  griddep_launch();
  extern __shared__ __align__(16) unsigned char smem[];
  const int nmel = a.n_mels;
  const float ref_db = 10.0f * log10f(a.ref);
  const bool lanes = a.mel_lane_ok != 0;
  unsigned char *sp = smem;
  float4 *tw4 = reinterpret_cast<float4 *>(sp);  // as frame_pair_kernel
  sp += size_t(16) * TPF * 16;
  float4 *win_s = reinterpret_cast<float4 *>(sp);
  sp += size_t(N) * 4;
  // real-split factors: row 2p + j0, column c holds those of c + 32 (4p + j0)
  // and c + 32 (4p + 2 + j0)
  float4 *rs_tw = reinterpret_cast<float4 *>(sp);
  sp += size_t(S::RS) * 16;
  float4 *wa_s = reinterpret_cast<float4 *>(sp);
  if (lanes) sp += size_t(16) * 16 * TPF;
  float2 *wb_s = reinterpret_cast<float2 *>(sp);
  if (lanes) sp += size_t(16) * 8 * TPF;
  int4 *lane_s = reinterpret_cast<int4 *>(sp);
  if (lanes) sp += size_t(16) * TPF;
  cpx2 *bufs = reinterpret_cast<cpx2 *>(sp);
  sp += size_t(np) * S::BS * 16;
  const int words = lanes ? nmel : a.mel_nnz;
  const bool staged = words <= S::MEL_SMEM_MAX;
  int *words_s = reinterpret_cast<int *>(sp);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int fp = warp >> 1;                // this warp's pair
  const int half = warp & 1;               // 0: even columns, 1: odd columns
  const int j = half * 32 + lane;          // stage-1 row, walk lane
  const int j0 = lane & 1;                 // stage-2 half of the column
  const int col = 2 * (lane >> 1) + half;  // stage-2 column k1
  const bool c0 = col == 0;
  const int partner = 2 * (half ? 15 - (lane >> 1) : (16 - (lane >> 1)) & 15) + (1 - j0);
  const float2 *twq = a.tw_split;  // W_N^t, t < N/4

  for (int i = tid; i < 16 * TPF; i += threads) {
    const int k = i / TPF, jj = i - k * TPF;
    const cpx u = root_q(twq, 2 * jj * k, N), w = root_q(twq, 2 * jj * (k + 16), N);
    tw4[i] = make_float4(u.x, u.y, w.x, w.y);
  }
  for (int i = tid; i < 16 * TPF; i += threads) {  // halved: see the header comment
    const int p = i / TPF, jj = i - p * TPF;
    const float2 u = __ldg(reinterpret_cast<const float2 *>(a.window) + jj + TPF * (2 * p));
    const float2 w = __ldg(reinterpret_cast<const float2 *>(a.window) + jj + TPF * (2 * p + 1));
    win_s[i] = make_float4(0.5f * u.x, 0.5f * u.y, 0.5f * w.x, 0.5f * w.y);
  }
  for (int i = tid; i < S::RS; i += threads) {
    const int row = i / 33, c = min(i - 33 * row, 31), p = row >> 1, jj0 = row & 1;  // (column 32 is padding)
    const float2 u = split_factors(root_q(twq, c + 32 * (4 * p + jj0), N), p < 4);
    const float2 w = split_factors(root_q(twq, c + 32 * (4 * p + 2 + jj0), N), p < 4);
    rs_tw[i] = make_float4(u.x, u.y, w.x, w.y);
  }
  bool twice = lanes && stage_walk<TPF>(a, wa_s, wb_s, lane_s, tid, threads);
  const int *src_words = lanes ? a.mel_band : reinterpret_cast<const int *>(a.mel_pw);
  if (staged)
    for (int i = tid; i < words; i += threads) words_s[i] = __ldg(src_words + i);
  const int *band = staged ? words_s : src_words;
  twice = __syncthreads_or(twice) != 0;
  griddep_wait();  // the tables are constant; the clips and their maxima are not
  if (fp >= np) return;  // a small batch: this warp only helped to stage the tables

  const WarpPairSync sync{fp};
  cpx2 *fb = bufs + fp * S::BS;
  f2 *P = reinterpret_cast<f2 *>(fb);
  cpx2 *parts = reinterpret_cast<cpx2 *>(P + PS * TPF);

  Units<S::UF, S::UT> units(a, fp, np);
  int vclip = -1;  // the clip vmax belongs to
  float vmax = -INFINITY;
  while (units.advance(a)) {  // uniform over the warp pair
    if (units.clip != vclip) {
      flush_max(a, vclip, vmax, lane);
      vclip = units.clip;
      vmax = -INFINITY;
    }
    const ClipDesc &cd = units.cd;
    const int t = units.first_frame();
    const bool vb = t + 1 < cd.n_frames;
    float *dst = a.out + (cd.frame_off + t) * (long long)nmel;

    cpx2 e[16], o[16];
    load_pair<TPF, D>(a, cd, t, j, win_s, e, o);
    {  // the samples that the next unit adds, into L1: one line a thread
      const long long at = (long long)(t + S::UF * np) * a.hop - a.pad + N - (S::UF - 1) * a.hop + j * 32;
      if (j * 32 < S::UF * a.hop && at >= 0 && at < cd.length)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.signal + cd.sig_off + at));
    }
    // ---- stage 1
    dft16(e);
    dft16(o);
    sync();  // the previous unit's reads of the buffer are done
    finish_stage1<TPF>(e, o, tw4 + j, [&](auto ki, cpx2 y) { fb[j * 33 + decltype(ki)::value] = y; });
    sync();
    // ---- stage 2a: 32-point DFT of rows j0 + 2 j1 of column col -> A_j0[q]
    cpx2 v[32];
#pragma unroll
    for (int j1 = 0; j1 < 32; j1++) v[j1] = fb[(j0 + 2 * j1) * 33 + col];
    dft32(v);
    // ---- stage 2b: combine the column's two halves; z[i] = Z[col + 32 (2i + j0)],
    // z[16 + i] = Z[col + 32 (2i + j0 + 32)]
    cpx2 z[32];
    static_for<0, 16>([&](auto ii) {
      constexpr int i = decltype(ii)::value;
      const cpx2 snd = csel(j0, v[2 * i], v[2 * i + 1]);
      const cpx2 rcv = {shfl2(snd.x, lane ^ 1), shfl2(snd.y, lane ^ 1)};
      const cpx2 ev = csel(j0, rcv, v[2 * i]);
      constexpr float ca = (float)ce_trig(2 * i, 64, 0), sa = -(float)ce_trig(2 * i, 64, 1);
      constexpr float cb = (float)ce_trig(2 * i + 1, 64, 0), sb = -(float)ce_trig(2 * i + 1, 64, 1);
      const cpx2 od = cmul(csel(j0, v[2 * i + 1], rcv), {j0 ? cb : ca, j0 ? sb : sa});
      z[i] = cadd(ev, od);
      z[16 + i] = csub(ev, od);
    });
    sync();  // every column is read: the buffer becomes P
    // ---- real split: pair i is (Z[k], Z[M - k]), k = col + 32 (2i + j0); the
    // partner's z[31 - i] holds Z[M - k] (column 0: this thread's own z)
    {
      f2 *Pa = P + col + PS * j0;                                       // bin col + 32 s at col + PS s
      f2 *Pb = P + (PS * (TPF - 1) + 32 - col - PS * j0) + (c0 ? 1 : 0);  // bin M - col - 32 s
      float4 rsp;
      cpx2 prev = z[0];
      static_for<0, 16>([&](auto ii) {
        constexpr int i = decltype(ii)::value;
        const cpx2 up = z[31 - i];
        const cpx2 rcv = {shfl2(up.x, partner), shfl2(up.y, partner)};
        const cpx2 zb = csel(c0, csel(j0, up, prev), rcv);
        prev = up;
        if constexpr (i % 2 == 0) rsp = rs_tw[(i + j0) * 33 + col];  // row 2 (i / 2) + j0
        f2 p, q;
        split_pair<(i < 8)>(z[i], zb, i % 2 == 0 ? rsp.x : rsp.z, i % 2 == 0 ? rsp.y : rsp.w, p, q);
        Pa[2 * PS * i] = p;
        if constexpr (i == 0) Pb[(c0 && !j0) ? -1 : 0] = q;  // column 0, s = 0: the Nyquist bin
        else Pb[-2 * PS * i] = q;
      });
      if (c0 && !j0) P[M / 2 + TPF / 2] = mul2(dup2(4.0f), fma2(prev.x, prev.x, mul2(prev.y, prev.y)));
    }
    sync();  // P complete

    // ---- log-mel rows of both frames + running clip max
    if (lanes) walk_bands<TPF>(a, sync, P, parts, j, {wa_s, wb_s, lane_s, band, twice}, ref_db, dst, true, vb, vmax);
    else row_bands<TPF>(a, sync, P, j, reinterpret_cast<const float *>(band), ref_db, dst, true, vb, vmax);
  }
  flush_max(a, vclip, vmax, lane);
}

static int sm_count_cached() {
  static std::atomic<int> cached[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev >= 0 && dev < 64 && (n = cached[dev].load()) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 148;
  if (dev >= 0 && dev < 64) cached[dev].store(n);
  return n;
}

// One CTA per SM, and as few of its warps (or warp pairs) at work as finish in
// the same number of rounds: a small batch spreads over all SMs (all warps
// stage the tables: a 3 s clip, one unit an SM, waits for nothing else).
// smem_of(w): shared memory with w workers.
template <typename K, typename Smem>
static cudaError_t launch_units(K kern, const FrontArgs &a, int per_tile, int workers, int threads, Smem smem_of,
                                int grid_limit, cudaStream_t s, int *launched) {
  int per_sm = 1, sms = sm_count_cached();
  if (grid_limit > 0 && sms > grid_limit) sms = grid_limit;
  const long long units = (long long)a.total_tiles * per_tile;
  const long long rounds = (units + (long long)sms * workers - 1) / ((long long)sms * workers);
  const int w = (int)((units + sms * rounds - 1) / (sms * rounds));
  const size_t smem = smem_of(w);
  int all = 0;
  cudaError_t e = persistent_geometry(reinterpret_cast<const void *>(kern), threads, smem, &per_sm, &all);
  if (e != cudaSuccess) return e;
  const long long grid = units < sms ? units : sms;
  if (grid < 1) return cudaSuccess;
  e = launch_after(kern, (unsigned)grid, threads, smem, s, a, w);
  if (e != cudaSuccess) return e;
  if (launched) *launched = (int)grid;
  return cudaGetLastError();
}

template <int LOG2N, int D>
static cudaError_t launch_pair_d(const FrontArgs &a, int grid_limit, cudaStream_t s, int *launched) {
  using S = PShape<LOG2N>;
  const int words = a.mel_lane_ok ? a.n_mels : a.mel_nnz;
  auto smem_of = [&](int w) {
    return pair_fixed_smem<LOG2N>() + (a.mel_lane_ok ? (16 * 24 + 16) * (size_t)S::TPF : 0) +
           w * pair_warp_smem<LOG2N>() + (words <= S::MEL_SMEM_MAX ? align16(4 * (size_t)words) : 0);
  };
  return launch_units(frame_pair_kernel<LOG2N, D>, a, S::UT, S::NW, 32 * S::NW, smem_of, grid_limit, s, launched);
}

template <int D>
static cudaError_t launch_pair4096_d(const FrontArgs &a, int grid_limit, cudaStream_t s, int *launched) {
  using S = P4Shape;
  const int words = a.mel_lane_ok ? a.n_mels : a.mel_nnz;
  auto smem_of = [&](int w) {
    return S::fixed + (a.mel_lane_ok ? S::walk : 0) + w * size_t(S::BS) * 16 +
           (words <= S::MEL_SMEM_MAX ? align16(4 * (size_t)words) : 0);
  };
  return launch_units(frame_pair4096_kernel<D>, a, S::UT, S::NP, 64 * S::NP, smem_of, grid_limit, s, launched);
}

// Shared gathers exist for the usual hops where they win, against D = 0 on 256
// clips of 15 s (whole step, us): n_fft/4 at n_fft 256 640 / 707, 512 483 / 515,
// 1024 451 / 461, 2048 413 / 427, 4096 513 / 535; n_fft/2 at 256 348 / 376, 512
// 265 / 278, 2048 227 / 234; 10 ms of 32 ms at 256 526 / 581, 512 402 / 426.  At n_fft
// 1024 neither of the last two does: 256 clips of 30 s 481 / 478 (n_fft/2) and
// 743 / 736 (10 ms of 32 ms), one clip 16.5 us in every form.
template <int LOG2N>
static cudaError_t launch_pair(const FrontArgs &a, int grid_limit, cudaStream_t s, int *launched) {
  constexpr int step = 2 * PShape<LOG2N>::TPF;  // samples per register step, n_fft / 32
  if (a.even_starts && a.hop == 8 * step) return launch_pair_d<LOG2N, 8>(a, grid_limit, s, launched);    // n_fft / 4
  if constexpr (LOG2N != 10)  // n_fft / 2
    if (a.even_starts && a.hop == 16 * step) return launch_pair_d<LOG2N, 16>(a, grid_limit, s, launched);
  if constexpr (LOG2N <= 9)  // 10 ms of a 32 ms frame: speech at 8 and 16 kHz
    if (a.even_starts && a.hop == 10 * step) return launch_pair_d<LOG2N, 10>(a, grid_limit, s, launched);
  return launch_pair_d<LOG2N, 0>(a, grid_limit, s, launched);
}

cudaError_t launch_frontend_pair(int log2n, const FrontArgs &a, int grid_limit, cudaStream_t s, int *launched) {
  switch (log2n) {
    case 8: return launch_pair<8>(a, grid_limit, s, launched);
    case 9: return launch_pair<9>(a, grid_limit, s, launched);
    case 10: return launch_pair<10>(a, grid_limit, s, launched);
    case 11: return launch_pair<11>(a, grid_limit, s, launched);
    case 12:
      if (a.hop == 1024 && a.even_starts) return launch_pair4096_d<8>(a, grid_limit, s, launched);
      return launch_pair4096_d<0>(a, grid_limit, s, launched);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace mm
