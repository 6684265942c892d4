"""The frame-pair kernels (launch variant 3, n_fft 256..4096): two frames at a
time, so the cases are the places where a pair can go wrong: one, two and
three frames, odd frame counts, clips shorter than a frame, edge pairs under
both paddings, the shared gather of hop n_fft/4 beside any other hop (odd
sample offsets among them), filterbanks whose bin pairs end two segments, one
segment or none, and the packed-row epilogue.

Bars: MFCC within 1e-4 of max |c| of the FP64 oracle, as every MFCC test; and
the log-mel rows within 2e-3 dB of the CTA-tile kernel's (variant 0) within
60 dB of the clip maximum, since each kernel is held to 1e-3 dB of the oracle
there."""

import numpy as np
import pytest

import metalmom_b200 as M
from metalmom_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MFCC_TOL = 1e-4
DB_TOL = 2e-3


def _device_floats(ptr, n):
    import torch

    class View:
        __cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False), "version": 2}

    return torch.as_tensor(View(), device="cuda").cpu().numpy().copy()


def _rows(variant, clips, n_mels, **params):
    """(MFCC, log-mel rows, clip maximum) per clip under a launch variant."""
    n_fft = params["n_fft"]
    old = M.tune_get(n_fft)
    M.tune_set(n_fft, variant)
    try:
        with M.Plan([len(c) for c in clips], n_mels=n_mels, n_mfcc=min(20, n_mels), **params) as plan:
            out = plan.execute_host(clips)
            return [(o, _device_floats(plan.clip_mel_db_ptr(i), plan.frames[i] * n_mels).reshape(-1, n_mels),
                     plan.clip_max_db(i)) if plan.frames[i] else (o, np.empty((0, n_mels)), 0.0)
                    for i, o in enumerate(out)]
    finally:
        M.tune_set(n_fft, old)


@pytest.mark.parametrize("pad", ["constant", "reflect"])
@pytest.mark.parametrize("n_fft,hop,n_mels", [
    (2048, 512, 128), (2048, 441, 128), (2048, 1024, 40), (2048, 512, 400), (2048, 512, 1100),
    (1024, 256, 64), (1024, 441, 128), (1024, 256, 260),
    (512, 128, 40), (512, 160, 80), (512, 128, 200),
    (256, 64, 40), (256, 85, 26), (256, 64, 120),
    (1024, 320, 64), (1024, 512, 128), (512, 256, 80), (256, 80, 40), (256, 128, 26),
    (4096, 1024, 128), (4096, 441, 64), (4096, 2048, 40), (4096, 1024, 900), (4096, 1024, 1100),
])
def test_pair_kernel_vs_cta_tile_kernel_and_oracle(n_fft, hop, n_mels, pad):
    sr = 22050
    lens = [n_fft + k * hop + d for k, d in ((0, 0), (1, 0), (2, 1), (7, 3), (8, 0), (61, 5))] + [n_fft // 2 + 1]
    clips = [synth.music_clip(n, sr, seed=n + n_mels) for n in lens]
    for center in (True, False):
        params = dict(sr=sr, n_fft=n_fft, hop_length=hop, center=center, pad_mode=pad)
        pair, tile = _rows(3, clips, n_mels, **params), _rows(0, clips, n_mels, **params)
        for y, (c, db, mx), (c0, db0, mx0) in zip(clips, pair, tile):
            assert c.shape == c0.shape and db.shape == db0.shape
            if not c.size:
                continue
            assert abs(mx - mx0) <= DB_TOL
            near = db0 >= mx0 - 60.0
            assert np.abs(db - db0)[near].max() <= DB_TOL, (len(y), center)
            if pad == "constant":
                exp = O.mfcc(y, sr, min(20, n_mels), n_fft, hop, n_fft, n_mels, center=center)
                assert O.mfcc_rel_error(c, exp) < MFCC_TOL, (len(y), center)


@pytest.mark.parametrize("n_fft,n_mels", [(2048, 128), (2048, 1100), (512, 40), (4096, 128), (4096, 1100)])
def test_pair_kernel_flags_only_the_frame_with_a_non_finite_sample(n_fft, n_mels):
    """A NaN reaches the frames that cover it and no other: the partner frame
    of a pair and its neighbours keep their values bit for bit."""
    sr, hop = 22050, n_fft // 4
    y = synth.music_clip(40 * hop, sr, seed=5)
    bad = y.copy()
    at = 20 * hop + 3
    bad[at] = np.nan
    params = dict(sr=sr, n_fft=n_fft, hop_length=hop)
    (_, clean, _), (_, got, _) = _rows(3, [y], n_mels, **params)[0], _rows(3, [bad], n_mels, **params)[0]
    t = np.arange(clean.shape[0])
    hit = (t * hop - n_fft // 2 <= at) & (at < t * hop + n_fft // 2)
    assert hit.any() and not hit.all()
    np.testing.assert_array_equal(got[~hit], clean[~hit])
    assert (got[hit] == got[hit][0, 0]).all() and got[hit][0, 0] == pytest.approx(-100.0, abs=1e-4)


def test_pair_kernel_small_and_large_batches_agree_bitwise():
    """The number of warps at work in a CTA follows the batch: the results do not."""
    clips = [synth.music_clip(20000 + 777 * i, 22050, seed=i) for i in range(60)]
    outs = M.mfcc_batch(clips * 4, sr=22050)
    for i in (0, 31, 59):
        one = M.mfcc_batch([clips[i]], sr=22050)[0]
        for k in range(4):
            np.testing.assert_array_equal(outs[i + 60 * k], one)
