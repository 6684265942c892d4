// Host runtime of libmetalmom.so (see runtime.h).
#include "runtime.h"

#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace mm {

int cuda_status(cudaError_t e) {
  switch (e) {
    case cudaSuccess: return MM_OK;
    case cudaErrorMemoryAllocation: return MM_ERR_ALLOC_FAILED;
    case cudaErrorNoDevice:
    case cudaErrorInsufficientDriver:
    case cudaErrorInvalidDevice: return MM_ERR_METAL_UNAVAILABLE;
    default: return MM_ERR_INTERNAL;
  }
}

int gpu_available() {
  static std::once_flag once;
  static int status = MM_ERR_METAL_UNAVAILABLE;
  std::call_once(once, [] {
    int n = 0;
    if (cudaGetDeviceCount(&n) == cudaSuccess && n > 0) status = MM_OK;
    else cudaGetLastError();
  });
  return status;
}

namespace {
// Launch variant per log2(n_fft) until mm_tune_set or mm_autotune stores
// another: variant 3 for n_fft 256..4096, 0 elsewhere; a mode without variant
// 3 falls back to 0.  Whole step against variant 0 on 64 clips of 30 s (hop
// n_fft/4): n_fft 256 323 / 520 us, 512 253 / 410, 1024 225 / 441, 2048 218 /
// 428, 4096 289 / 449; on one clip of 1 to 30 s between equal and 1.5x faster
// (n_fft 256 and 512 with few frames: within one 2 us step either way).
std::atomic<int> g_tuned[16] = {0, 0, 0, 0, 0, 0, 0, 0, kWarpVariant, kWarpVariant, kWarpVariant, kWarpVariant,
                                kWarpVariant, 0, 0, 0};
}

int tuned_variant(int log2n) { return (log2n >= 0 && log2n < 16) ? g_tuned[log2n].load() : 0; }
void set_tuned_variant(int log2n, int v) {
  if (log2n >= 0 && log2n < 16) g_tuned[log2n].store(v);
}
int group_variant(const Group &g) {
  if (g.dft_form != DFT_FFT_F32) return kDftVariant;
  const int nv = frame_variants(g.log2n, g.mode, g.power == 2.0f);
  const int v = tuned_variant(g.log2n);
  if (v == kTcVariant)  // the tensor-core kernel: n_fft 2048 on the MFCC path only
    return (g.log2n == 11 && g.mode == MODE_MELDB && g.power == 2.0f) ? kTcVariant : (nv > kWarpVariant ? kWarpVariant : 0);
  return (v >= 0 && v < nv) ? v : 0;
}

int is_pow2(long long n) { return n > 0 && (n & (n - 1)) == 0; }
int ilog2(long long n) {
  int l = 0;
  while ((1LL << l) < n) l++;
  return l;
}

long long frame_count(long long length, int n_fft, int hop, int center) {
  const long long padded = center ? length + 2LL * (n_fft / 2) : length;
  if (padded < n_fft || !is_pow2(n_fft) || hop <= 0) return 0;
  return 1 + (padded - n_fft) / hop;
}

bool same_group(const Group &a, const Group &b) {
  return std::tie(a.mode, a.sr, a.n_fft, a.hop, a.win, a.window_zero, a.center, a.pad_mode, a.n_mels,
                  a.n_mfcc_eff, a.fmin, a.fmax, a.top_db, a.power, a.amin, a.ref, a.dft_form, a.post, a.lag) ==
         std::tie(b.mode, b.sr, b.n_fft, b.hop, b.win, b.window_zero, b.center, b.pad_mode, b.n_mels,
                  b.n_mfcc_eff, b.fmin, b.fmax, b.top_db, b.power, b.amin, b.ref, b.dft_form, b.post, b.lag);
}

int output_rows(const Group &g) {
  switch (g.mode) {
    case MODE_SPECTRUM: return g.n_fft / 2 + 1;
    case MODE_COMPLEX: return 2 * (g.n_fft / 2 + 1);  // interleaved (re, im) per bin
    case MODE_MEL: return g.n_mels;
    default: return g.post == POST_ONSET_MEAN ? 1 : (g.post == POST_ONSET_BANDS ? g.n_mels : g.n_mfcc_eff);
  }
}

// ---------------------------------------------------------------------------
// resident tables
// ---------------------------------------------------------------------------
namespace {
struct TableKey {
  int dev, sr, n_fft, win, window_zero, n_mels, n_mfcc;
  float fmin, fmax;
  int dft;  // 1: also the DFT-as-GEMM basis
  bool operator<(const TableKey &o) const {
    return std::tie(dev, sr, n_fft, win, window_zero, n_mels, n_mfcc, fmin, fmax, dft) <
           std::tie(o.dev, o.sr, o.n_fft, o.win, o.window_zero, o.n_mels, o.n_mfcc, o.fmin, o.fmax, o.dft);
  }
};
std::mutex g_table_mu;
std::map<TableKey, DevTables *> g_tables;
}  // namespace

const DevTables *get_tables(const Group &g, int *status) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    *status = cuda_status(e);
    return nullptr;
  }
  const int n_mels = mode_has_mel(g.mode) ? g.n_mels : 0;
  const int n_mfcc = (g.mode == MODE_MELDB) ? g.n_mfcc_eff : 0;
  // basis images: none (FFT), bf16 (the two bf16 forms) or fp16 (the fp16-split form)
  const int basis_kind = g.dft_form == DFT_GEMM_F16X3 ? 2 : (g.dft_form != DFT_FFT_F32 ? 1 : 0);
  TableKey k{dev, g.sr, g.n_fft, g.win, g.window_zero, n_mels, n_mfcc, g.fmin, g.fmax, basis_kind};
  std::lock_guard<std::mutex> lock(g_table_mu);
  auto it = g_tables.find(k);
  if (it != g_tables.end()) {
    *status = MM_OK;
    return it->second;
  }
  DevTables *t = new DevTables();
  cudaStream_t s;
  e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) {
    e = build_tables(*t, g.sr, g.n_fft, g.win, n_mels, g.fmin, g.fmax, n_mfcc, g.window_zero, s);
    // the error word of the group's kernels with bounded waits (tensor-core
    // DFT forms and frame kernel)
    if (e == cudaSuccess) e = cudaMalloc(&t->dft_err, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemsetAsync(t->dft_err, 0, sizeof(unsigned), s);
    if (e == cudaSuccess && g.dft_form != DFT_FFT_F32) {
      t->dft = dft_shape(g.n_fft, g.win);
      e = cudaMalloc(&t->dft_basis, dft_basis_bytes(t->dft));
      if (e == cudaSuccess)
        e = build_dft_basis(t->dft_basis, t->dft, g.win, g.window_zero, g.dft_form == DFT_GEMM_F16X3, s);
    }
    cudaError_t e2 = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = e2;
    cudaStreamDestroy(s);
  }
  if (e != cudaSuccess) {
    *status = cuda_status(e);
    cudaFree(t->window);
    cudaFree(t->tw_stage);
    cudaFree(t->tw_split);
    cudaFree(t->tw_tiny);
    cudaFree(t->mel_w);
    cudaFree(t->mel_pw);
    cudaFree(t->mel_info);
    cudaFree(t->mel_w2);
    cudaFree(t->mel_seg);
    cudaFree(t->mel_lw);
    cudaFree(t->mel_lane);
    cudaFree(t->mel_band);
    cudaFree(t->dct);
    cudaFree(t->dft_basis);
    cudaFree(t->dft_err);
    delete t;
    return nullptr;
  }
  g_tables[k] = t;
  *status = MM_OK;
  return t;
}

// ---------------------------------------------------------------------------
// batch layout
// ---------------------------------------------------------------------------
static inline long long round_up(long long v, long long a) { return (v + a - 1) / a * a; }

void make_layout(const Group &g, const int64_t *lengths, int n, Layout &L) {
  L.clips.resize(n);
  L.tile_clip.clear();
  L.dct_tile_clip.clear();
  L.dct_tile_first.clear();
  L.F = frames_per_tile(g.log2n, g.variant);
  const int rows = output_rows(g);
  long long sig = 0, frames = 0, out = 0;
  int tiles = 0;
  for (int i = 0; i < n; i++) {
    ClipDesc &c = L.clips[i];
    const long long T = frame_count(lengths[i], g.n_fft, g.hop, g.center);
    c.sig_off = sig;
    c.length = lengths[i];
    c.frame_off = frames;
    c.out_off = out;
    c.n_frames = (int)T;
    c.tile_base = tiles;
    const int nt = (int)((T + L.F - 1) / L.F);
    for (int q = 0; q < nt; q++) L.tile_clip.push_back(i);
    tiles += nt;
    if (g.mode == MODE_MELDB)
      for (long long f = 0; f < T; f += kDctTile) {
        L.dct_tile_clip.push_back(i);
        L.dct_tile_first.push_back((int)f);
      }
    sig = round_up(sig + lengths[i], 4);
    frames += T;
    out += (long long)rows * T;
  }
  L.sig_elems = sig;
  L.total_frames = frames;
  L.out_elems = out;
  L.meldb_elems = (g.mode == MODE_MELDB) ? frames * (long long)g.n_mels : 0;
  L.scale_elems = (g.mode == MODE_MELDB && g.dft_form == DFT_GEMM_F16X3) ? frames : 0;
}

namespace {
struct Offsets {
  size_t signal, clips, tile_clip, dct_clip, dct_first, desc_end, clip_max, meldb, out, scale, total;
};
Offsets offsets(const Layout &L) {
  Offsets o;
  const size_t n = L.clips.size();
  size_t p = 0;
  o.signal = p;
  p = round_up(p + sizeof(float) * (size_t)L.sig_elems, 256);
  o.clips = p;
  p = round_up(p + sizeof(ClipDesc) * n, 16);
  o.tile_clip = p;
  p = round_up(p + sizeof(int) * L.tile_clip.size(), 16);
  o.dct_clip = p;
  p = round_up(p + sizeof(int) * L.dct_tile_clip.size(), 16);
  o.dct_first = p;
  p = round_up(p + sizeof(int) * L.dct_tile_first.size(), 16);
  o.desc_end = p;
  p = round_up(p, 256);
  o.clip_max = p;
  p = round_up(p + sizeof(unsigned) * (n > 0 ? n : 1), 256);
  o.meldb = p;
  p = round_up(p + sizeof(float) * (size_t)L.meldb_elems, 256);
  o.out = p;
  p = round_up(p + sizeof(float) * (size_t)L.out_elems, 256);
  o.scale = p;
  p = round_up(p + sizeof(float) * (size_t)L.scale_elems, 256);
  o.total = p;
  return o;
}
}  // namespace

size_t arena_bytes(const Group &, const Layout &L) { return offsets(L).total; }

size_t carve_arena(const Group &, const Layout &L, char *base, DevBatch &b) {
  const Offsets o = offsets(L);
  b.signal = reinterpret_cast<float *>(base + o.signal);
  b.clips = reinterpret_cast<ClipDesc *>(base + o.clips);
  b.tile_clip = reinterpret_cast<int *>(base + o.tile_clip);
  b.dct_tile_clip = reinterpret_cast<int *>(base + o.dct_clip);
  b.dct_tile_first = reinterpret_cast<int *>(base + o.dct_first);
  b.clip_max = reinterpret_cast<unsigned *>(base + o.clip_max);
  b.meldb = reinterpret_cast<float *>(base + o.meldb);
  b.out = reinterpret_cast<float *>(base + o.out);
  b.frame_scale = L.scale_elems > 0 ? reinterpret_cast<float *>(base + o.scale) : nullptr;
  return o.desc_end - o.clips;
}

void pack_descriptors(const Layout &L, char *host) {
  // host mirrors the arena from the clips segment on
  const Offsets o = offsets(L);
  if (!L.clips.empty()) memcpy(host, L.clips.data(), sizeof(ClipDesc) * L.clips.size());
  if (!L.tile_clip.empty())
    memcpy(host + (o.tile_clip - o.clips), L.tile_clip.data(), sizeof(int) * L.tile_clip.size());
  if (!L.dct_tile_clip.empty())
    memcpy(host + (o.dct_clip - o.clips), L.dct_tile_clip.data(), sizeof(int) * L.dct_tile_clip.size());
  if (!L.dct_tile_first.empty())
    memcpy(host + (o.dct_first - o.clips), L.dct_tile_first.data(), sizeof(int) * L.dct_tile_first.size());
}

int take_error_word(const Group &g, const DevTables *t) {
  if (!t || !t->dft_err || (g.dft_form == DFT_FFT_F32 && g.variant != kTcVariant)) return MM_OK;
  unsigned flag = 0;
  cudaError_t e = cudaMemcpy(&flag, t->dft_err, sizeof(unsigned), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_status(e);
  if (!flag) return MM_OK;
  cudaMemset(t->dft_err, 0, sizeof(unsigned));
  return MM_ERR_INTERNAL;
}

cudaError_t enqueue_batch(const Group &g, const Layout &L, const DevTables *t, const DevBatch &b,
                          cudaStream_t s, cudaEvent_t *ev, int *n_launches) {
  cudaError_t e;
  int launches = 0;
  if (ev && (e = cudaEventRecord(ev[0], s)) != cudaSuccess) return e;
  const int n = (int)L.clips.size();
  if (g.mode == MODE_MELDB) {
    if ((e = launch_fill_u32(b.clip_max, encode_max_init(), n, s)) != cudaSuccess) return e;
    launches++;
  }
  if (ev && (e = cudaEventRecord(ev[1], s)) != cudaSuccess) return e;
  FrontArgs a;
  a.signal = b.signal;
  a.clips = b.clips;
  a.tile_clip = b.tile_clip;
  a.total_tiles = (int)L.tile_clip.size();
  a.hop = g.hop;
  a.pad = g.center ? g.n_fft / 2 : 0;
  a.pad_mode = g.pad_mode;
  a.window = t->window;
  a.tw_stage = t->tw_stage;
  a.tw_split = t->tw_split;
  a.tw_tiny = t->tw_tiny;
  a.mel_info = t->mel_info;
  a.mel_pw = t->mel_pw;
  a.mel_nnz = t->mel_nnz;
  a.mel_w2 = t->mel_w2;
  a.mel_seg = t->mel_seg;
  a.mel_seg_ok = t->mel_seg_ok;
  a.mel_lw = t->mel_lw;
  a.mel_lane = t->mel_lane;
  a.mel_band = t->mel_band;
  a.mel_lane_ok = t->mel_lane_ok;
  a.n_mels = mode_has_mel(g.mode) ? g.n_mels : 0;
  a.power = g.power;
  a.amin = g.amin;
  a.ref = g.ref;
  a.out = (g.mode == MODE_MELDB) ? b.meldb : b.out;
  a.clip_max = b.clip_max;
  a.err = t->dft_err;
  a.even_starts = 1;  // make_layout puts every clip at a multiple of 4 samples
  int grid = 0;
  if (g.dft_form == DFT_GEMM_F16X3 && g.mode == MODE_MELDB) {
    a.frame_scale = b.frame_scale;
    if ((e = launch_frame_scale(a, t->dft, s)) != cudaSuccess) return e;
    launches++;
  }
  if (g.dft_form != DFT_FFT_F32 && g.mode == MODE_MELDB)
    e = launch_dft_gemm(g.dft_form, a, t->dft, t->dft_basis, t->dft_err, s, &grid);
  else
    e = launch_frontend(g.log2n, g.mode, g.variant, a, 0, s, &grid);
  if (e != cudaSuccess) return e;
  if (grid > 0) launches++;
  if (ev && (e = cudaEventRecord(ev[2], s)) != cudaSuccess) return e;
  if (g.mode == MODE_MELDB && g.post != POST_DCT && !L.dct_tile_clip.empty()) {
    OnsetArgs o;
    o.mel_db = b.meldb;
    o.clips = b.clips;
    o.tile_clip = b.dct_tile_clip;
    o.tile_first = b.dct_tile_first;
    o.total_tiles = (int)L.dct_tile_clip.size();
    o.clip_max = b.clip_max;
    o.n_mels = g.n_mels;
    o.lag = g.lag;
    o.shift = g.lag + (g.center ? g.n_fft / (2 * g.hop) : 0);
    o.bands = g.post == POST_ONSET_BANDS;
    o.top_db = g.top_db;
    o.out = b.out;
    if ((e = launch_onset(o, s)) != cudaSuccess) return e;
    launches++;
  } else if (g.mode == MODE_MELDB && g.n_mfcc_eff > 0 && !L.dct_tile_clip.empty()) {
    DctArgs d;
    d.mel_db = b.meldb;
    d.clips = b.clips;
    d.tile_clip = b.dct_tile_clip;
    d.tile_first = b.dct_tile_first;
    d.total_tiles = (int)L.dct_tile_clip.size();
    d.clip_max = b.clip_max;
    d.basis = t->dct;
    d.n_mels = g.n_mels;
    d.n_mfcc = g.n_mfcc_eff;
    d.top_db = g.top_db;
    d.out = b.out;
    if ((e = launch_dct(d, s)) != cudaSuccess) return e;
    launches++;
  }
  if (ev && (e = cudaEventRecord(ev[3], s)) != cudaSuccess) return e;
  if (n_launches) *n_launches = launches;
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// per-thread workspace
// ---------------------------------------------------------------------------
namespace {
struct WorkspaceHolder {
  Workspace ws;
  ~WorkspaceHolder() {
    // Process teardown may already have destroyed the CUDA context; ignore errors.
    if (ws.stream) cudaStreamDestroy(ws.stream);
    for (cudaEvent_t e : ws.piece)
      if (e) cudaEventDestroy(e);
    if (ws.dev) cudaFree(ws.dev);
    if (ws.host) cudaFreeHost(ws.host);
  }
};
thread_local WorkspaceHolder t_ws;
}  // namespace

int thread_workspace(size_t dev_bytes, size_t host_bytes, Workspace **out) {
  Workspace &w = t_ws.ws;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_status(e);
  if (w.device != dev) {
    // First use on this thread, or the caller switched devices: start over.
    if (w.stream) {
      cudaStreamSynchronize(w.stream);
      cudaStreamDestroy(w.stream);
      w.stream = nullptr;
    }
    for (cudaEvent_t &p : w.piece) {
      if (p) cudaEventDestroy(p);
      p = nullptr;
    }
    if (w.dev) cudaFree(w.dev);  // unified addressing: frees on its own device
    w.dev = nullptr;
    w.dev_bytes = 0;
    e = cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking);
    for (cudaEvent_t &p : w.piece)
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p, cudaEventDisableTiming);
    if (e != cudaSuccess) return cuda_status(e);
    w.device = dev;
  }
  if (dev_bytes > w.dev_bytes) {
    cudaStreamSynchronize(w.stream);
    if (w.dev) cudaFree(w.dev);
    w.dev = nullptr;
    w.dev_bytes = 0;
    const size_t want = dev_bytes + dev_bytes / 4;
    e = cudaMalloc(&w.dev, want);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return MM_ERR_ALLOC_FAILED;
    }
    w.dev_bytes = want;
  }
  if (host_bytes > w.host_bytes) {
    cudaStreamSynchronize(w.stream);
    if (w.host) cudaFreeHost(w.host);
    w.host = nullptr;
    w.host_bytes = 0;
    const size_t want = host_bytes + host_bytes / 4;
    e = cudaMallocHost(&w.host, want);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return MM_ERR_ALLOC_FAILED;
    }
    w.host_bytes = want;
  }
  *out = &w;
  return MM_OK;
}

// ---------------------------------------------------------------------------
// host results
// ---------------------------------------------------------------------------
// Staging of a result on its way into pageable memory (see fetch_staged).
constexpr size_t kFetchPiece = size_t(512) << 10, kFetchSlots = sizeof(Workspace::piece) / sizeof(cudaEvent_t);

// Through the staging in pieces, each copied on to `r` while the next ones cross
// the bus.  Into memory that has been touched before, 5.3 MB / 2.6 MB / 0.66 MB
// take 342 / 179 / 46 us; the whole result staged first 398 / 205 / 47, a copy by
// the driver into the pageable memory itself 287 / 158 / 58 but, where the
// pages are new, 2 409 / 1 200 / 321 against 1 441 / 733 / 187.  Pieces of 256 KB
// 365 / 189 / 45, of 1 MB 334 / 179 / 47.  Measured and left out: non-temporal
// stores (311 / 165 / 56), three threads sharing the pieces (209 / 121 / 50, but
// 90th percentiles of 670 / 430 / 72 against 354 / 186 / 48).
static cudaError_t fetch_staged(const float *d, size_t bytes, Workspace *ws, float *r) {
  constexpr size_t kPiece = kFetchPiece, kSlots = kFetchSlots;
  const char *src = reinterpret_cast<const char *>(d);
  char *dst = reinterpret_cast<char *>(r);
  const size_t pieces = (bytes + kPiece - 1) / kPiece;
  if (pieces <= 1) {
    cudaError_t e = cudaMemcpyAsync(ws->host, src, bytes, cudaMemcpyDeviceToHost, ws->stream);
    const cudaError_t e2 = cudaStreamSynchronize(ws->stream);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) memcpy(dst, ws->host, bytes);
    return e;
  }
  auto size = [&](size_t i) { return std::min(kPiece, bytes - i * kPiece); };
  auto issue = [&](size_t i) {
    const cudaError_t e = cudaMemcpyAsync(ws->host + (i % kSlots) * kPiece, src + i * kPiece, size(i),
                                          cudaMemcpyDeviceToHost, ws->stream);
    return e == cudaSuccess ? cudaEventRecord(ws->piece[i % kSlots], ws->stream) : e;
  };
  cudaError_t e = cudaSuccess;
  for (size_t i = 0; i < pieces && i < kSlots && e == cudaSuccess; i++) e = issue(i);
  for (size_t i = 0; i < pieces && e == cudaSuccess; i++) {
    if ((e = cudaEventSynchronize(ws->piece[i % kSlots])) != cudaSuccess) break;
    memcpy(dst + i * kPiece, ws->host + (i % kSlots) * kPiece, size(i));
    if (i + kSlots < pieces) e = issue(i + kSlots);
  }
  if (e != cudaSuccess) cudaStreamSynchronize(ws->stream);  // the last piece's event stands for the stream otherwise
  return e;
}

int fetch_result(const float *d, size_t bytes, const ResultPlace &place, Workspace *ws, float **out) {
  Workspace *same = nullptr;  // waits for the stream if the staging has to grow
  const int st = thread_workspace(0, std::min(bytes, kFetchPiece * kFetchSlots), &same);
  if (st != MM_OK) return st;
  const bool given = place.dst && place.dst_bytes == bytes;
  float *r = given ? place.dst : static_cast<float *>(malloc(bytes));
  if (!r) return MM_ERR_ALLOC_FAILED;
  const cudaError_t e = fetch_staged(d, bytes, ws, r);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (!given) free(r);
    return cuda_status(e);
  }
  *out = r;
  return MM_OK;
}

cudaError_t upload(float *d, const float *h, size_t bytes, Workspace *ws) {
  if (bytes >= kDirectUpload) return cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, ws->stream);
  memcpy(ws->host, h, bytes);
  return cudaMemcpyAsync(d, ws->host, bytes, cudaMemcpyHostToDevice, ws->stream);
}

void fill_buffer(MMBuffer *out, float *data, long long rows, long long cols) {
  out->data = data;
  for (int i = 0; i < 8; i++) out->shape[i] = 0;
  out->shape[0] = rows;
  out->shape[1] = cols;
  out->ndim = 2;
  out->dtype = 0;
  out->count = rows * cols;
}

}  // namespace mm
