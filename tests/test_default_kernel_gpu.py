"""The kernel that runs unless another is chosen: n_fft 256..4096 on the MFCC
path is the frame-pair kernel (launch variant 3), also after a launch choice has
been read, changed and set back; and what holds of its default size holds of
every size it has."""

import numpy as np
import pytest

import metalmom_b200 as M
from goldens import golden, signal_440
from metalmom_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SR = 22050
SIZES = [256, 512, 1024, 2048, 4096]
MFCC_TOL = 1e-4  # of max |c|, as every MFCC test


@pytest.fixture
def variant():
    """Set a size's variant for the test."""
    old = {n: M.tune_get(n) for n in SIZES}

    def choose(n_fft, v):
        M.tune_set(n_fft, v)

    yield choose
    for n, v in old.items():
        M.tune_set(n, v)


@pytest.mark.parametrize("n_fft", [256, 512, 1024])
def test_the_default_survives_saving_and_restoring(n_fft, variant):
    y = synth.music_clip(2 * SR + 11, SR, seed=n_fft)

    def run():
        return M.mfcc(y, sr=SR, n_fft=n_fft, hop_length=n_fft // 4, n_mels=40)

    variant(n_fft, 3)
    pair = run()
    variant(n_fft, 0)
    tile = run()
    assert not np.array_equal(pair, tile)  # or the check below would show nothing
    fresh = _own_process(n_fft)
    np.testing.assert_array_equal(fresh, pair)


def _own_process(n_fft):
    """The same call in a process that has only read, set and set back."""
    import os
    import subprocess
    import sys
    import tempfile
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "c.npy")
        code = (f"import numpy as np, metalmom_b200 as M\nfrom metalmom_b200 import synth\n"
                f"old = M.tune_get({n_fft})\nM.tune_set({n_fft}, 2)\nM.tune_set({n_fft}, old)\n"
                f"y = synth.music_clip({2 * SR + 11}, {SR}, seed={n_fft})\n"
                f"np.save({path!r}, M.mfcc(y, sr={SR}, n_fft={n_fft}, hop_length={n_fft // 4}, n_mels=40))\n")
        subprocess.run([sys.executable, "-c", code], cwd=root, check=True, timeout=300)
        return np.load(path)


@pytest.mark.parametrize("n_fft", SIZES)
@pytest.mark.parametrize("part", [4, 5])  # hop n_fft/4: shared gather; n_fft/5: any hop
def test_small_and_large_batches_agree_bitwise(n_fft, part, variant):
    """The number of warps at work in a CTA follows the batch: the results do not."""
    variant(n_fft, 3)
    clips = [synth.music_clip(6 * n_fft + 777 * i, SR, seed=i) for i in range(60)]
    params = dict(sr=SR, n_fft=n_fft, hop_length=n_fft // part, n_mels=40)
    outs = M.mfcc_batch(clips * 4, **params)
    for i in (0, 31, 59):
        one = M.mfcc_batch([clips[i]], **params)[0]
        for k in range(4):
            np.testing.assert_array_equal(outs[i + 60 * k], one)


def test_the_reference_golden_at_1024(variant):
    variant(1024, 3)
    got = M.mfcc(y=signal_440(), sr=SR, n_mfcc=13, n_fft=1024, n_mels=40)
    np.testing.assert_allclose(got, golden("mfcc_440hz_13_1024"), rtol=1e-4, atol=1e-4)

@pytest.mark.parametrize("center", [True, False])
@pytest.mark.parametrize("n_fft,hop,n_mels", [
    (256, 64, 40), (256, 80, 40), (256, 85, 26), (256, 128, 26), (512, 128, 40), (512, 160, 80), (512, 256, 80),
    (1024, 256, 64), (1024, 320, 64), (1024, 441, 64), (1024, 512, 64), (2048, 512, 128), (2048, 441, 128),
    (2048, 1024, 40), (4096, 1024, 128), (4096, 441, 64), (4096, 2048, 40),
])
def test_reflected_edges_vs_oracle(n_fft, hop, n_mels, center, variant):
    """Both edges of clips from just over the padding (one reflection) to many
    frames, odd lengths among them."""
    variant(n_fft, 3)
    lens = [n_fft // 2 + 1, n_fft, n_fft + hop, 2 * n_fft + 3, n_fft + 7 * hop + 1]
    clips = [synth.music_clip(n, SR, seed=n + hop) for n in lens]
    params = dict(sr=SR, n_fft=n_fft, hop_length=hop, n_mels=n_mels, center=center, pad_mode="reflect")
    for y, got in zip(clips, M.mfcc_batch(clips, **params)):
        exp = O.mfcc(y, SR, min(20, n_mels), n_fft, hop, n_fft, n_mels, center=center, pad_mode=O.PAD_REFLECT)
        assert got.shape == exp.shape, len(y)
        if exp.size:
            assert O.mfcc_rel_error(got, exp) < MFCC_TOL, (len(y), O.mfcc_rel_error(got, exp))
