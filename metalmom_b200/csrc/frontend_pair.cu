// Frame-pair front-end kernel (launch variant 3, n_fft 256..2048, MFCC path):
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
//
// Only warp-level synchronisation is used.  The window is staged in shared
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
// the kernel now waits on its own latencies (issue 44 %, shared-memory pipe
// 67 %).  256 clips of 30 s at n_fft 2048, hop 512, 128 bands: 0.90 -> 0.77 ms
// (whole step 0.954 -> 0.833); 512 clips of 10 s at n_fft 512, hop 160, 80
// bands: 0.46 ms against 0.62 for the CTA-tile kernel (whole step 0.431).
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
  static constexpr int PS = 34;  // float pairs per 32 bins of the spectrum
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

int warp_frames_per_tile(int log2n) {
  switch (log2n) {
    case 8: return PShape<8>::F;
    case 9: return PShape<9>::F;
    case 10: return PShape<10>::F;
    case 11: return PShape<11>::F;
    case 12: return 8;  // frame_warp2_kernel: one frame per warp pair, 16 warps
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
  return k + 2 * (q < TPF - 1 ? q : TPF - 1);
}

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
      // W = c - i s: both entries of p lie on the same side of an eighth of a turn
      rs_tw[i] = p < 4 ? make_float4(u.x, -u.y / u.x, w.x, -w.y / w.x)
                       : make_float4(-u.y, u.x / -u.y, -w.y, w.x / -w.y);
    }
  bool twice = false;  // some pair of bins ends two segments
  if (lanes) {
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
      // {first | second segment ends by pair, first part's byte offset, parts
      // the head takes over from the next lanes, the empty segments' slot}
      lane_s[i] = make_int4((int)(m1 | m2 << 16), 16 * (w.y & 1023), (w.y >> 10) & 63, w.y >> 16);
      if (m2) twice = true;
    }
    for (int i = tid; i < 16 * TPF; i += threads) {
      const int g = i / TPF, j = i - g * TPF;
      const bool fa = flush_bit(__ldg(a.mel_lane + j), 2 * g) != 0;
      const float2 u = __ldg(a.mel_lw + 2 * g * TPF + j), w = __ldg(a.mel_lw + (2 * g + 1) * TPF + j);
      wa_s[i] = make_float4(u.x, u.y, fa ? 0.0f : w.x, fa ? 0.0f : w.y);
      wb_s[i] = make_float2(fa ? w.x : 0.0f, fa ? w.y : 0.0f);
    }
  }
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
  const unsigned gmask = (TPF == 32) ? FULL : (((1u << TPF) - 1u) << (grp * TPF));

  // This CTA's units (2 FPW consecutive frames of one clip each) are a
  // contiguous range dealt to its warps in turn, so that the samples its
  // warps read at a time overlap.
  const long long total = (long long)a.total_tiles * S::UT;
  const int u_end = (int)((blockIdx.x + 1) * total / gridDim.x);
  int cur = -1, next_clip = -1;  // next_clip: first unit past the current clip
  ClipDesc cd{};
  int vclip = -1;  // the clip vmax belongs to
  float vmax = -INFINITY;

  // Moves on to this warp's next unit with a frame in it; false at the end.
  int u = (int)(blockIdx.x * total / gridDim.x) + warp - nw;
  auto advance = [&]() {
    while ((u += nw) < u_end) {
      if (u >= next_clip) {  // warp-uniform: every frame of a tile belongs to one clip
        cur = __ldg(a.tile_clip + u / S::UT);
        cd = load_clip(a.clips + cur);
        next_clip = (cd.tile_base + (cd.n_frames + S::F - 1) / S::F) * S::UT;
      }
      if ((u - cd.tile_base * S::UT) * S::UF < cd.n_frames) return true;
    }
    return false;
  };
  auto first_frame = [&]() { return (u - cd.tile_base * S::UT) * S::UF + 2 * grp; };

  // Raw samples (x[2n], x[2n+1]), n = l + TPF r, of this warp's next unit:
  // register r of frame t, and with D > 0 of frame t + 1 at r + D.
  constexpr int Q = D > 0 ? 32 + D : 32;
  auto gather_frame = [&](auto &dst_q, int t, int reach) {
    constexpr int n = sizeof(dst_q) / sizeof(float2);
    const long long s0 = (long long)t * a.hop - a.pad;
    const float *base = a.signal + cd.sig_off + s0 + 2 * l;
    if (s0 >= 0 && s0 + reach + N <= cd.length) {
      if (D > 0 || ((cd.sig_off + s0) & 1) == 0) {
#pragma unroll
        for (int r = 0; r < n; r++) dst_q[r] = __ldg(reinterpret_cast<const float2 *>(base + 2 * TPF * r));
      } else {
#pragma unroll
        for (int r = 0; r < n; r++)
          dst_q[r] = make_float2(__ldg(base + 2 * TPF * r), __ldg(base + 2 * TPF * r + 1));
      }
    } else {  // frames that reach into the padding (a few per clip)
      float2 te[n];
      gather_edge_n<n>(te, a.signal + cd.sig_off, s0 + 2 * l, cd.length, a.pad_mode, 2 * TPF);
#pragma unroll
      for (int r = 0; r < n; r++) dst_q[r] = te[r];
    }
  };
  // window; even registers into e, odd ones into o
  auto window = [&](const float2 *qa, const float2 *qb, cpx2 *e, cpx2 *o) {
    const float4 *wb = win_s + l;
#pragma unroll
    for (int r = 0; r < 32; r += 2) {
      const float4 w = wb[TPF * (r / 2)];
      e[r / 2] = {pk2(qa[r].x * w.x, qb[r].x * w.x), pk2(qa[r].y * w.y, qb[r].y * w.y)};
      o[r / 2] = {pk2(qa[r + 1].x * w.z, qb[r + 1].x * w.z), pk2(qa[r + 1].y * w.w, qb[r + 1].y * w.w)};
    }
  };

  bool more = advance();
  while (more) {
    if (cur != vclip) {
      float m = vmax;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
      if (lane == 0 && vclip >= 0 && m > -INFINITY) atomicMax(a.clip_max + vclip, enc_f(m));
      vclip = cur;
      vmax = -INFINITY;
    }
    const int tw0 = first_frame() - 2 * grp, t = tw0 + 2 * grp;
    const bool va = t < cd.n_frames, vb = t + 1 < cd.n_frames;
    float *dst = a.out + (cd.frame_off + t) * (long long)nmel;

    cpx2 e[16], o[16];
    {
      float2 q[Q];
      gather_frame(q, t, D > 0 ? a.hop : 0);
      if constexpr (D > 0) {
        window(q, q + D, e, o);
      } else {
        float2 qb[32];
        gather_frame(qb, t + 1, 0);
        window(q, qb, e, o);
      }
    }
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
      static_for<0, 16>([&](auto ki) {
        constexpr int k = decltype(ki)::value;
        using R = Rot<k, 32>;
        cpx2 lo, hi;
        rot_butterfly<R>(e[k], R::rot(o[k]), lo, hi);
        const float4 tk = tw4[k * TPF + l];
        if constexpr (k > 0) lo = cmul(lo, {tk.x, tk.y});
        hi = cmul(hi, {tk.z, tk.w});
        if constexpr (TPF == 32) {
          row[(k & 8) + ((k & 7) ^ (l & 7))] = lo;
          row[16 + (k & 8) + ((k & 7) ^ (l & 7))] = hi;
        } else {
          row[k] = lo;
          row[k + 16] = hi;
        }
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
        const f2 ex = add2(za.x, zb.x), ey = sub2(za.y, zb.y);
        const f2 ox = add2(za.y, zb.y), oy = sub2(zb.x, za.x);
        if constexpr (i % 2 == 0) rsp = rs_tw[32 * (i / 2) + l];
        const f2 sc = dup2(i % 2 == 0 ? rsp.x : rsp.z), rt = dup2(i % 2 == 0 ? rsp.y : rsp.w);
        f2 wr, wi;  // W_N^(l + 32 i) O without its scale
        if constexpr (i < 8) {
          wr = fma2(oy, rt, ox);
          wi = fma2(neg2(ox), rt, oy);
        } else {
          wr = fma2(ox, rt, oy);
          wi = fma2(oy, rt, neg2(ox));
        }
        const f2 xr = fma2(wr, sc, ex), xi = fma2(wi, sc, ey);
        const f2 yr = fma2(neg2(wr), sc, ex), yi = fma2(neg2(wi), sc, ey);
        const f2 p = fma2(xr, xr, mul2(xi, xi)), q = fma2(yr, yr, mul2(yi, yi));
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

    more = advance();

    // ---- log-mel rows of both frames + running clip max
    if (lanes) {
      // Lane l sums its 32 bins (the last lane also the Nyquist bin) into
      // (R, F) = (rising, falling weight) times P and stores the sums in the
      // next part slot at every segment end.  Bins go in pairs: the second
      // bin of a pair has its weights in one of two sets, zero in the other,
      // (wa.z, wa.w) for the segment that the first bin belongs to and wb for
      // a segment that it starts, so one predicated store and restart serve
      // a pair wherever in it the segment ends.  Pairs that end two segments
      // (bands of a single bin) take the second end in a branch of their own.
      const int4 li = lane_s[l];
      const unsigned fl = (unsigned)li.x;
      const uint32_t part0 = smem_u32(parts);
      uint32_t at = part0 + (unsigned)li.y;  // the next part's slot
      const float4 *pl = reinterpret_cast<const float4 *>(P + PS * l);
      const float4 *wa = wa_s + l;
      const float2 *wb = wb_s + l;
      const f2 zero = dup2(0.0f);
      f2 R = zero, Fs = zero;
      // the frames' non-finite check: the largest bit pattern of a power (a
      // power is never negative; NaN and inf lie at or above inf's pattern)
      unsigned mxa = 0u, mxb = 0u;
      static_for<0, 16>([&](auto gi) {
        constexpr int g = decltype(gi)::value;
        const float4 pq = pl[g], u = wa[g * TPF];
        const float2 w = wb[g * TPF];
        mxa = max(max(mxa, __float_as_uint(pq.x)), __float_as_uint(pq.z));
        mxb = max(max(mxb, __float_as_uint(pq.y)), __float_as_uint(pq.w));
        const f2 p0 = pk2(pq.x, pq.y), p1 = pk2(pq.z, pq.w);
        R = fma2(p0, dup2(u.x), R);
        Fs = fma2(p0, dup2(u.y), Fs);
        R = fma2(p1, dup2(u.z), R);
        Fs = fma2(p1, dup2(u.w), Fs);
        walk_end<g>(p1, w.x, w.y, fl, R, Fs, at);
        if (twice && (fl & (0x10000u << g))) {
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
        const float4 pq = pl[16];
        const float2 w = __ldg(a.mel_lw + 32 * TPF + l);
        mxa = max(mxa, __float_as_uint(pq.x));
        mxb = max(mxb, __float_as_uint(pq.y));
        R = fma2(pk2(pq.x, pq.y), dup2(w.x), R);
        Fs = fma2(pk2(pq.x, pq.y), dup2(w.y), Fs);
      }
      walk_store(at, R, Fs);
      if (l == 0) parts[li.w] = {zero, zero};  // the empty segments' slot
      const unsigned ba = __ballot_sync(FULL, mxa >= 0x7f800000u), bb = __ballot_sync(FULL, mxb >= 0x7f800000u);
      // added to a frame's band sums: NaN where a bin of it is not finite
      const f2 nan2 = pk2((ba & gmask) ? __int_as_float(0x7fc00000) : 0.0f, (bb & gmask) ? __int_as_float(0x7fc00000) : 0.0f);
      __syncwarp();
      // a lane whose last part heads a segment adds the parts of the lanes the
      // segment runs into
      if (li.z) {
        cpx2 *h = parts + ((at - part0) >> 4);
        cpx2 hv = *h;
        for (int j = 1; j <= li.z; j++) hv = cadd(hv, h[j]);
        *h = hv;
      }
      __syncwarp();
      // band m is the head of segment m (rising) plus the head of segment
      // m + 1 (falling); four bands at a time, so that their reads overlap.
      // The lane tables hold finite weights only: no band is NaN by itself.
      const char *pb = reinterpret_cast<const char *>(parts);
      for (int m0 = l; m0 < nmel; m0 += 4 * TPF) {
        int bw[4];
        f2 acc[4];
#pragma unroll
        for (int i = 0; i < 4; i++) bw[i] = m0 + i * TPF < nmel ? band[m0 + i * TPF] : 0;
#pragma unroll
        for (int i = 0; i < 4; i++)
          acc[i] = add2(*reinterpret_cast<const f2 *>(pb + 16 * (bw[i] & 4095)),
                        *reinterpret_cast<const f2 *>(pb + 8 + 16 * ((bw[i] >> 12) & 4095)));
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int m = m0 + i * TPF;
          float xa, xb;
          un2(add2(acc[i], nan2), xa, xb);
          const float da = fmaf(k10Log10of2, __log2f(fmaxf(xa, a.amin)), -ref_db);
          const float db = fmaf(k10Log10of2, __log2f(fmaxf(xb, a.amin)), -ref_db);
          if (va && m < nmel) {
            dst[m] = da;
            vmax = fmaxf(vmax, da);
          }
          if (vb && m < nmel) {
            dst[nmel + m] = db;
            vmax = fmaxf(vmax, db);
          }
        }
      }
    } else {
      unsigned mxa = 0u, mxb = 0u;  // the non-finite check: this lane's share of the bins
      for (int k = l; k <= M; k += TPF) {
        float pa, pb;
        un2(P[pair_bin<TPF>(k)], pa, pb);
        mxa = max(mxa, __float_as_uint(pa));
        mxb = max(mxb, __float_as_uint(pb));
      }
      const bool bada = (__ballot_sync(FULL, mxa >= 0x7f800000u) & gmask) != 0;
      const bool badb = (__ballot_sync(FULL, mxb >= 0x7f800000u) & gmask) != 0;
      for (int m = l; m < nmel; m += TPF) {
        const int4 info = __ldg(a.mel_info + m);
        const float *wr = melw + info.z;
        f2 acc = dup2(0.0f);
        for (int q = 0; q < info.y; q++) acc = fma2(P[pair_bin<TPF>(info.x + q)], dup2(wr[q]), acc);
        float xa, xb;
        un2(acc, xa, xb);
        if (info.w || bada) xa = __int_as_float(0x7fc00000);
        if (info.w || badb) xb = __int_as_float(0x7fc00000);
        if (va) {
          const float val = db10_frame(xa, a.amin, ref_db);
          dst[m] = val;
          vmax = fmaxf(vmax, val);
        }
        if (vb) {
          const float val = db10_frame(xb, a.amin, ref_db);
          dst[nmel + m] = val;
          vmax = fmaxf(vmax, val);
        }
      }
    }
  }
  float m = vmax;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
  if (lane == 0 && vclip >= 0 && m > -INFINITY) atomicMax(a.clip_max + vclip, enc_f(m));
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

template <int LOG2N, int D>
static cudaError_t launch_pair_d(const FrontArgs &a, int grid_limit, cudaStream_t s, int *launched) {
  using S = PShape<LOG2N>;
  int per_sm = 1, sms = sm_count_cached();
  if (grid_limit > 0 && sms > grid_limit) sms = grid_limit;
  // One CTA per SM, and as few of its warps at work as finish in the same
  // number of rounds: a small batch spreads over all SMs (all warps stage the
  // tables: a 3 s clip, one unit an SM, waits for nothing else).
  const long long units = (long long)a.total_tiles * S::UT;
  const long long rounds = (units + (long long)sms * S::NW - 1) / ((long long)sms * S::NW);
  const int nw = (int)((units + sms * rounds - 1) / (sms * rounds));
  const int words = a.mel_lane_ok ? a.n_mels : a.mel_nnz;
  const size_t smem = pair_fixed_smem<LOG2N>() + (a.mel_lane_ok ? (16 * 24 + 16) * (size_t)S::TPF : 0) +
                      nw * pair_warp_smem<LOG2N>() + (words <= S::MEL_SMEM_MAX ? align16(4 * (size_t)words) : 0);
  auto kern = frame_pair_kernel<LOG2N, D>;
  cudaError_t e = persistent_geometry(reinterpret_cast<const void *>(kern), 32 * S::NW, smem, &per_sm, &sms);
  if (e != cudaSuccess) return e;
  long long grid = sms;
  if (grid_limit > 0 && grid > grid_limit) grid = grid_limit;
  if (grid > units) grid = units;
  if (grid < 1) return cudaSuccess;
  e = launch_after(kern, (unsigned)grid, 32 * S::NW, smem, s, a, nw);
  if (e != cudaSuccess) return e;
  if (launched) *launched = (int)grid;
  return cudaGetLastError();
}

template <int LOG2N>
static cudaError_t launch_pair(const FrontArgs &a, int grid_limit, cudaStream_t s, int *launched) {
  constexpr int step = 2 * PShape<LOG2N>::TPF;  // samples per register step
  if (a.hop == 8 * step && a.even_starts) return launch_pair_d<LOG2N, 8>(a, grid_limit, s, launched);    // n_fft / 4
  return launch_pair_d<LOG2N, 0>(a, grid_limit, s, launched);
}

cudaError_t launch_frontend_pair(int log2n, const FrontArgs &a, int grid_limit, cudaStream_t s, int *launched) {
  switch (log2n) {
    case 8: return launch_pair<8>(a, grid_limit, s, launched);
    case 9: return launch_pair<9>(a, grid_limit, s, launched);
    case 10: return launch_pair<10>(a, grid_limit, s, launched);
    case 11: return launch_pair<11>(a, grid_limit, s, launched);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace mm
