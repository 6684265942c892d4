"""The work that programs built on this package have it do, as timed cases.

Every case goes through the package's public entry points (``metalmom_b200``).
Two kinds of program are stood for:

* one-off calls on host arrays, the functions that MetalMom's own Python
  package has (``mfcc``, ``melspectrogram``, ``stft``, ``istft``) and the
  batched form of the first (``mfcc_batch``): audio comes from a decoder as a
  NumPy array and the features go on as one, so the whole call counts;
* feature extraction over a corpus or inside a training loop, where the audio
  is already on the device and a ``Plan`` is kept and replayed, and decibel
  scaling of a spectrogram that another program holds as a CUDA tensor.

Parameter sets are the ones of the benchmark's workloads (music: 22.05 kHz,
n_fft 2048, hop 512, 128 bands, 20 coefficients; speech: 16 kHz, n_fft 512,
window 400, hop 160, 80 bands, 13 coefficients; the uneven batch's groups).
Launch variants are the defaults: nothing is autotuned.

``exact`` restates the path in float64 with torch alone.
"""

import math

import numpy as np
import torch

import metalmom_b200 as M

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
MUSIC = dict(sr=22050, n_fft=2048, hop=512, win=2048, n_mels=128, n_mfcc=20, fmin=0.0, fmax=0.0,
             center=True, reflect=False)
SPEECH = dict(sr=16000, n_fft=512, hop=160, win=400, n_mels=80, n_mfcc=13, fmin=20.0, fmax=8000.0,
              center=True, reflect=False)
HIRES = dict(MUSIC, sr=44100, n_fft=4096, hop=1024, win=4096)
EVENTS = dict(sr=44100, n_fft=1024, hop=441, win=882, n_mels=64, n_mfcc=13, fmin=50.0, fmax=16000.0,
              center=True, reflect=True)


def listed():
    return [
        # one MFCC call on a short clip of odd length (a keyword, a sample): latency
        dict(MUSIC, name="mfcc_call_3s", kind="mfcc", samples=64007),
        # the default MFCC call on a 30 s excerpt
        dict(MUSIC, name="mfcc_call_30s", kind="mfcc", samples=661500),
        # the default mel spectrogram of the same excerpt (a network's input, a picture)
        dict(MUSIC, name="mel_call_30s", kind="mel", samples=661500),
        # magnitude spectrogram of 30 s: the widest result of the path
        dict(MUSIC, name="stft_call_30s", kind="stft", samples=661500),
        # the way back: a masked complex spectrogram to audio (separation, denoising)
        dict(MUSIC, name="istft_call_30s", kind="istft", samples=661500),
        # one batched call on ragged recordings with a 10 ms hop at 44.1 kHz, short window, reflected edges
        dict(EVENTS, name="batch_call_ragged", kind="batch", clips=40, samples=300007, ragged=True),
        # decibels of a resident power spectrogram relative to its maximum
        dict(name="db_device", kind="db", rows=128, frames=330752, ref_max=True, top_db=80.0),
        # one resident 30 s clip at a time: the smallest replay, launches and latency
        dict(MUSIC, name="plan_one_30s", kind="plan", clips=1, samples=661500, ragged=False),
        # the benchmark's batch: 256 excerpts of 30 s
        dict(MUSIC, name="plan_music_256", kind="plan", clips=256, samples=661500, ragged=False),
        # the speech front end over 512 utterances of 10 s
        dict(SPEECH, name="plan_speech_512", kind="plan", clips=512, samples=160000, ragged=False),
        # the long transform at 44.1 kHz
        dict(HIRES, name="plan_hires_64", kind="plan", clips=64, samples=1323000, ragged=False),
        # clips of 1 to 120 s, each with its own parameters (12 groups): an uncurated archive
        dict(name="plan_mixed_160", kind="mixed", clips=160, low_s=1.0, high_s=120.0),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _draw_params(rng):
    kind = rng.randrange(4)
    if kind == 0:
        return dict(SPEECH, n_mels=rng.choice([40, 64, 80]), n_mfcc=rng.choice([13, 20]))
    if kind == 1:
        return dict(EVENTS, hop=rng.choice([441, 220, 512]), win=rng.choice([882, 1024]),
                    reflect=rng.random() < 0.5, n_mels=rng.choice([40, 64, 96, 128]))
    n_fft = rng.choice([256, 512, 1024, 2048, 2048, 4096])
    return dict(MUSIC, sr=rng.choice([22050, 44100]), n_fft=n_fft, win=n_fft,
                hop=rng.choice([n_fft // 4, n_fft // 4, n_fft // 2]),
                n_mels=rng.choice([40, 64, 128]) if n_fft > 512 else 40,
                n_mfcc=rng.choice([13, 20, 20, 40]), center=rng.random() < 0.8)


def draw(rng):
    kind = rng.choice(["mfcc", "mel", "stft", "istft", "batch", "db", "plan", "plan", "plan", "mixed"])
    if kind == "db":
        return dict(kind="db", rows=rng.choice([40, 64, 80, 128, 1025]), frames=_log_int(rng, 100, 40000),
                    ref_max=rng.random() < 0.5, top_db=rng.choice([80.0, 80.0, 60.0]))
    if kind == "mixed":
        return dict(kind="mixed", clips=_log_int(rng, 12, 140), low_s=1.0, high_s=float(rng.randrange(10, 120)))
    p = _draw_params(rng)
    if kind == "batch":
        return dict(p, kind="batch", clips=_log_int(rng, 2, 60), samples=_log_int(rng, 16000, 300000) | 1, ragged=True)
    if kind == "plan":
        clips = _log_int(rng, 1, 256)
        return dict(p, kind="plan", clips=clips, samples=_log_int(rng, 16000, min(2000000, 100000000 // clips)),
                    ragged=rng.random() < 0.5)
    if kind == "stft" or kind == "istft":
        p = dict(MUSIC, n_fft=rng.choice([512, 1024, 2048, 4096]))
        p.update(win=p["n_fft"], hop=p["n_fft"] // 4)
    return dict(p, kind=kind, samples=_log_int(rng, 16000, 2000000), reflect=False)  # the one-clip calls pad with zeros


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _audio(n, sr, seed):
    """Seeded music-like audio on the device: a few partials under a slow
    envelope, decaying clicks and a noise floor, clipped to [-1, 1]."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed)
    h = np.random.default_rng(seed)
    t = torch.arange(n, device=dev, dtype=torch.float64) / sr
    y = torch.zeros(n, device=dev, dtype=torch.float64)
    for _ in range(int(h.integers(2, 6))):
        f, a, ph = h.uniform(50.0, 0.45 * sr), h.uniform(0.05, 0.4), h.uniform(0.0, 2.0 * np.pi)
        y += a * torch.sin(2.0 * np.pi * f * t + ph)
    y *= 0.55 + 0.45 * torch.sin(2.0 * np.pi * h.uniform(0.1, 4.0) * t)
    y += 0.01 * torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    decay = 0.5 * torch.exp(-torch.arange(1600, device=dev, dtype=torch.float64) / 200.0)
    for pos in h.integers(0, n, 8):
        m = min(1600, n - int(pos))
        y[int(pos):int(pos) + m] += decay[:m]
    return y.clamp_(-1.0, 1.0).float()


def _lengths(case, seed):
    """Lengths belong to the case, not to the seed: a plan is kept and its audio changes."""
    n = case["clips"]
    if case["kind"] == "mixed":
        h = np.random.default_rng(2024)
        return [int(h.uniform(case["low_s"], case["high_s"]) * _mixed_params(n)[i]["sr"]) for i in range(n)]
    if not case["ragged"]:
        return [case["samples"]] * n
    h = np.random.default_rng(77)
    return [max(8192, int(case["samples"] * h.uniform(0.2, 1.0))) for _ in range(n)]


def _mixed_params(n):
    """The uneven batch's groups, dealt over the clips."""
    h = np.random.default_rng(2025)
    out = []
    for _ in range(n):
        n_fft = int(h.choice([1024, 2048, 4096]))
        out.append(dict(MUSIC, sr=int(h.choice([22050, 44100])), n_fft=n_fft, win=n_fft, hop=n_fft // 4,
                        n_mels=int(h.choice([64, 128]))))
    return out


def _keywords(p):
    """A parameter set as keywords of the batched entry points."""
    return dict(sr=p["sr"], n_fft=p["n_fft"], hop_length=p["hop"], win_length=p["win"], center=p["center"],
                pad_mode="reflect" if p["reflect"] else "constant", n_mels=p["n_mels"], n_mfcc=p["n_mfcc"],
                fmin=p["fmin"], fmax=p["fmax"] if p["fmax"] > 0.0 else None)


def _clips(case, seed):
    """(lengths, parameters per clip, audio per clip) of a batch."""
    lens = _lengths(case, seed)
    params = _mixed_params(case["clips"]) if case["kind"] == "mixed" else [case] * case["clips"]
    return lens, params, (_audio(n, p["sr"], seed * 4096 + i) for i, (n, p) in enumerate(zip(lens, params)))


def _masked_spectrum(case, seed):
    """A complex spectrogram as a separation program hands it back: the STFT
    of audio times a mask in [0, 1] (complex64, on the device)."""
    y = _audio(case["samples"], case["sr"], seed)
    n_fft, hop = case["n_fft"], case["hop"]
    w = torch.hann_window(n_fft, periodic=True, dtype=torch.float32, device=y.device)
    S = torch.stft(y, n_fft, hop, n_fft, w, center=True, pad_mode="constant", return_complex=True)
    g = torch.Generator(device=y.device).manual_seed(seed + 9)
    return S * torch.rand(S.shape, generator=g, device=y.device)


def _spectrogram(case, seed):
    """Power values over the dynamic range of music: log-normal, with silent frames."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed)
    x = torch.randn(case["rows"], case["frames"], generator=g, device=dev)
    x = torch.exp(3.0 * x - 2.0)
    x[:, torch.rand(case["frames"], generator=g, device=dev) < 0.02] = 0.0
    return x


class _Floats:
    """A float32 range of a plan's device memory, for torch.as_tensor; the
    tensor holds this object, and so the plan that owns the memory."""

    def __init__(self, plan, address, count):
        self.plan = plan
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (address, False), "version": 2}


def _device_floats(plan, address, count):
    return torch.as_tensor(_Floats(plan, address, count), device="cuda")


def _output_runs(plan):
    """(offset, count) of the plan's results, clips that follow each other in one run."""
    spans = sorted((plan.out_offsets[i], plan.clip_rows[i] * plan.frames[i]) for i in range(plan.n))
    runs = []
    for off, cnt in spans:
        if runs and runs[-1][0] + runs[-1][1] == off:
            runs[-1][1] += cnt
        else:
            runs.append([off, cnt])
    return runs


_streams = {}


def _work_stream():
    """The program's own stream: its replays follow each other on it."""
    d = torch.cuda.current_device()
    if d not in _streams:
        _streams[d] = torch.cuda.Stream()
    return _streams[d]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "db":
        return {"kind": kind, "x": _spectrogram(case, seed), "ref": np.max if case["ref_max"] else 1.0,
                "top_db": case["top_db"]}
    if kind == "istft":
        return {"kind": kind, "case": case, "S": _masked_spectrum(case, seed).cpu().numpy()}
    if kind in ("mfcc", "mel", "stft"):
        return {"kind": kind, "case": case, "y": _audio(case["samples"], case["sr"], seed).cpu().numpy()}
    lens, params, audio = _clips(case, seed)
    if kind == "batch":
        return {"kind": kind, "clips": [y.cpu().numpy() for y in audio], "keywords": _keywords(case)}
    if kind == "mixed":
        plan = M.Plan(lens, clip_params=[_keywords(p) for p in params])
    else:
        plan = M.Plan(lens, **_keywords(case))
    for i, y in enumerate(audio):
        _device_floats(plan, plan.device_input + 4 * plan.in_offsets[i], lens[i]).copy_(y)
    out = [_device_floats(plan, plan.device_output + 4 * off, cnt) for off, cnt in _output_runs(plan)]
    torch.cuda.synchronize()
    return {"kind": kind, "plan": plan, "out": out, "stream": _work_stream().cuda_stream}


def run(state):
    kind = state["kind"]
    if kind in ("plan", "mixed"):
        state["plan"].execute(stream=state["stream"])
        return state["out"]
    if kind == "db":
        return M.power_to_db_device(state["x"], ref=state["ref"], top_db=state["top_db"])
    if kind == "batch":
        return M.mfcc_batch(state["clips"], **state["keywords"])
    c = state["case"]
    if kind == "stft":
        return M.stft(state["y"], n_fft=c["n_fft"], hop_length=c["hop"], win_length=c["win"], center=c["center"])
    if kind == "istft":
        return M.istft(state["S"], hop_length=c["hop"], win_length=c["win"], length=c["samples"])
    fmax = c["fmax"] if c["fmax"] > 0.0 else None
    if kind == "mel":
        return M.melspectrogram(state["y"], sr=c["sr"], n_fft=c["n_fft"], hop_length=c["hop"], win_length=c["win"],
                                center=c["center"], n_mels=c["n_mels"], fmin=c["fmin"], fmax=fmax)
    return M.mfcc(state["y"], sr=c["sr"], n_mfcc=c["n_mfcc"], n_fft=c["n_fft"], hop_length=c["hop"],
                  win_length=c["win"], n_mels=c["n_mels"], fmin=c["fmin"], fmax=fmax, center=c["center"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _frames(n, p):
    padded = n + 2 * (p["n_fft"] // 2) if p["center"] else n
    return 0 if padded < p["n_fft"] else 1 + (padded - p["n_fft"]) // p["hop"]


def _fft_flops(n_fft):
    return 2.5 * n_fft * math.log2(n_fft)


def work(case):
    kind = case["kind"]
    if kind == "db":
        n = case["rows"] * case["frames"]
        return {"bytes": 8.0 * n, "flops": 4.0 * n}
    if kind in ("batch", "plan", "mixed"):
        lens = _lengths(case, 0)
        params = _mixed_params(case["clips"]) if kind == "mixed" else [case] * case["clips"]
    else:
        lens, params = [case["samples"]], [case]
    total_b = total_f = 0.0
    for n, p in zip(lens, params):
        T, bins = _frames(n, p), p["n_fft"] // 2 + 1
        if kind == "stft":
            b, f = 4.0 * (n + bins * T), T * (_fft_flops(p["n_fft"]) + 4 * bins)
        elif kind == "istft":
            b, f = 4.0 * (2 * bins * T + n), T * (_fft_flops(p["n_fft"]) + 2 * p["n_fft"])
        else:
            rows = p["n_mels"] if kind == "mel" else min(p["n_mfcc"], p["n_mels"])
            b = 4.0 * (n + rows * T)
            f = T * (_fft_flops(p["n_fft"]) + 7 * bins)
            if kind != "mel":
                f += T * 2.0 * rows * p["n_mels"]
        total_b += b
        total_f += f
    return {"bytes": total_b, "flops": total_f}


# ---------------------------------------------------------------------------
# the same in float64
# ---------------------------------------------------------------------------
def _window64(n_fft, win, dev):
    w = torch.zeros(n_fft, dtype=torch.float64, device=dev)
    k = torch.arange(win, dtype=torch.float64, device=dev)
    off = (n_fft - win) // 2
    w[off:off + win] = 0.5 - 0.5 * torch.cos(2.0 * np.pi * k / win)
    return w


def _spectrum64(y, p):
    """rfft of every frame, [frames, bins], in blocks."""
    n_fft, pad = p["n_fft"], p["n_fft"] // 2
    y = y.double()
    if p["center"]:
        mode = "reflect" if p["reflect"] else "constant"
        y = torch.nn.functional.pad(y[None, None], (pad, pad), mode=mode)[0, 0]
    fr = y.unfold(0, n_fft, p["hop"])
    w = _window64(n_fft, p["win"], y.device)
    for i in range(0, fr.shape[0], 16384):
        yield torch.fft.rfft(fr[i:i + 16384] * w)


def _mel_weights64(p, dev):
    """Slaney filterbank [n_mels, bins]."""
    def to_mel(f):
        return f * 3.0 / 200.0 if f < 1000.0 else 15.0 + math.log(f / 1000.0) / (math.log(6.4) / 27.0)

    def to_hz(m):
        return np.where(m < 15.0, m * 200.0 / 3.0, 1000.0 * np.exp((m - 15.0) * (math.log(6.4) / 27.0)))

    fmax = p["fmax"] if p["fmax"] > 0.0 else p["sr"] / 2.0
    e = to_hz(np.linspace(to_mel(p["fmin"]), to_mel(fmax), p["n_mels"] + 2))
    f = np.arange(p["n_fft"] // 2 + 1) * p["sr"] / p["n_fft"]
    up = (f[None] - e[:-2, None]) / (e[1:-1] - e[:-2])[:, None]
    down = (e[2:, None] - f[None]) / (e[2:] - e[1:-1])[:, None]
    W = np.maximum(0.0, np.minimum(up, down)) * (2.0 / (e[2:] - e[:-2]))[:, None]
    return torch.from_numpy(W).to(dev)


def _mel64(y, p):
    W = _mel_weights64(p, y.device)
    return torch.cat([(X.real.square() + X.imag.square()) @ W.T for X in _spectrum64(y, p)])  # [frames, mels]


def _mfcc64(y, p):
    db = 10.0 * torch.log10(_mel64(y, p).clamp_min(float(np.float32(1e-10))))
    db = torch.maximum(db, db.max() - 80.0)
    N, K = p["n_mels"], min(p["n_mfcc"], p["n_mels"])
    n = torch.arange(N, dtype=torch.float64, device=y.device)
    k = torch.arange(K, dtype=torch.float64, device=y.device)
    B = torch.cos(np.pi * k[:, None] * (2.0 * n[None] + 1.0) / (2.0 * N)) * math.sqrt(2.0 / N)
    B[0] *= math.sqrt(0.5)
    return B @ db.T


def _istft64(S, case):
    n_fft, hop, n = case["n_fft"], case["hop"], case["samples"]
    w = _window64(n_fft, case["win"], S.device)
    fr = torch.fft.irfft(S.to(torch.complex128).T, n_fft) * w
    total = n_fft + (fr.shape[0] - 1) * hop
    y = torch.zeros(total, dtype=torch.float64, device=S.device)
    ws = torch.zeros_like(y)
    at = (torch.arange(fr.shape[0], device=S.device)[:, None] * hop + torch.arange(n_fft, device=S.device)).reshape(-1)
    y.index_add_(0, at, fr.reshape(-1))
    ws.index_add_(0, at, w.square().repeat(fr.shape[0]))
    y = torch.where(ws > 1e-10, y / ws, y)[n_fft // 2:]
    out = torch.zeros(n, dtype=torch.float64, device=S.device)
    m = min(n, y.numel())
    out[:m] = y[:m]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "db":
        x = _spectrogram(case, seed).double()
        ref = x.max() if case["ref_max"] else 1.0
        db = 10.0 * torch.log10(x.clamp_min(float(np.float32(1e-10))) / ref)
        return torch.maximum(db, db.max() - case["top_db"])
    if kind == "istft":
        return _istft64(_masked_spectrum(case, seed), case)
    if kind in ("mfcc", "mel", "stft"):
        y = _audio(case["samples"], case["sr"], seed)
        if kind == "mfcc":
            return _mfcc64(y, case)
        if kind == "mel":
            return _mel64(y, case).T.contiguous()
        return torch.cat([X.abs() for X in _spectrum64(y, case)]).T.contiguous()
    lens, params, audio = _clips(case, seed)
    each = [_mfcc64(y, p) for y, p in zip(audio, params)]
    if kind == "batch":
        return each
    if kind == "plan":
        return [torch.cat([c.reshape(-1) for c in each])]
    # a mixed plan keeps the clips of one parameter set together, sets in order of first appearance
    groups = {}
    for c, p in zip(each, params):
        groups.setdefault(tuple(sorted(p.items())), []).append(c.reshape(-1))
    return [torch.cat(g) for g in groups.values()]
