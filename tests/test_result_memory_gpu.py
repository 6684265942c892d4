"""Whose memory a result lies in.  The one-clip calls return ordinary arrays:
pageable, owned by NumPy, and left alone by later calls whatever the caller has
still queued on them.  ``mm_init_into`` writes a result of the announced size
to the caller's memory and mallocs any other."""

import numpy as np
import pytest

import metalmom_b200 as M
from metalmom_b200._bridge import OWN_BYTES
from metalmom_b200._native import ffi, lib

pytestmark = pytest.mark.gpu


def _clip(seed, n=300000):
    return (0.3 * np.random.default_rng(seed).standard_normal(n)).astype(np.float32)


def _calls():
    """Every call that returns a large result, by name."""
    y, S = _clip(1), np.abs(M.stft(_clip(2)))
    X = M.stft_complex(_clip(3))
    return {
        "stft": lambda: M.stft(y), "stft uncentred": lambda: M.stft(y, n_fft=512, hop_length=100, center=False),
        "stft_complex": lambda: M.stft_complex(y), "istft": lambda: M.istft(X),
        "istft length": lambda: M.istft(X, length=123457), "istft uncentred": lambda: M.istft(X, center=False),
        "melspectrogram": lambda: M.melspectrogram(y), "mel of S": lambda: M.melspectrogram(S=S),
        "mfcc": lambda: M.mfcc(y, n_mfcc=128), "mfcc of S": lambda: M.mfcc(S=S, n_mfcc=900),
        "power_to_db": lambda: M.power_to_db(S), "amplitude_to_db": lambda: M.amplitude_to_db(S),
        "delta": lambda: M.delta(S), "stack_memory": lambda: M.stack_memory(S[:200], n_steps=3),
        "onset": lambda: M.onset_strength(y, aggregate=False), "onset 1-D": lambda: M.onset_strength(_clip(4, 70000), hop_length=1),
    }


def test_results_are_pageable_and_do_not_change_under_a_queued_copy():
    """A non-blocking upload of a result that is dropped at once, behind a long
    kernel: the calls that follow must not write into what it still reads."""
    import torch
    y = [_clip(i) for i in range(4)]
    want = [M.stft(v).copy() for v in y]
    assert want[0].nbytes >= OWN_BYTES
    assert not torch.from_numpy(M.stft(y[0])).is_pinned()
    s = torch.cuda.Stream()
    got = []
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)  # about 50 ms
        for v in y:
            got.append(torch.from_numpy(M.stft(v)).to("cuda", non_blocking=True))
    for v in y:
        M.stft(v)
    s.synchronize()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy(), w)


def test_large_results_can_be_resized_as_small_ones():
    for y in (_clip(1, 3000), _clip(1)):
        a = M.stft(y)
        assert a.flags.owndata and a.flags.writeable and a.flags.c_contiguous
        first = a.ravel()[:50].copy()
        a.resize((5, 10), refcheck=False)
        np.testing.assert_array_equal(a.ravel(), first)


def test_results_come_in_the_announced_memory(monkeypatch):
    """The direct route is the one that runs, and gives what the other gives."""
    import metalmom_b200._bridge as B
    taken = []
    plain = B.take_buffer
    monkeypatch.setattr(B, "take_buffer", lambda buf: (taken.append(1), plain(buf))[1])
    calls = _calls()
    taken.clear()
    direct = {k: f() for k, f in calls.items()}
    assert not taken
    monkeypatch.setattr(B, "_empty", lambda shape: None)
    for k, f in calls.items():
        other = f()
        assert direct[k].nbytes >= OWN_BYTES and direct[k].shape == other.shape, k
        np.testing.assert_array_equal(direct[k], other, err_msg=k)
    assert len(taken) == len(calls)


PIECE = (512 << 10) // 4


@pytest.mark.parametrize("count", [1, 65536] + [k * PIECE + d for k in (1, 2, 4, 5, 9) for d in (-1, 0, 1)])
def test_staging_pieces(count):
    """Sizes around the staging's pieces and slots (512 KB x 4), written to the
    destination where the size is the announced one and to malloc where not."""
    x = np.random.default_rng(count).uniform(0.5, 2.0, count).astype(np.float32)
    p = ffi.cast("const float*", x.ctypes.data)
    for announced in (count, count + 1):
        dst = np.full(count + 1, 7.0, np.float32)
        at = ffi.cast("float*", dst.ctypes.data)
        ctx = lib.mm_init_into(at, announced)
        out = ffi.new("MMBuffer*")
        assert lib.mm_stack_memory(ctx, p, count, 1, count, 1, 1, out) == 0  # one step: a copy
        lib.mm_destroy(ctx)
        if announced == count:
            assert out.data == at and dst[count] == 7.0
            got = dst[:count]
        else:
            assert out.data != at and (dst == 7.0).all()
            got = np.frombuffer(ffi.buffer(out.data, 4 * count), np.float32).copy()
            lib.mm_buffer_free(out)
        np.testing.assert_array_equal(got, x)


def test_a_refused_destination():
    x = np.zeros(4, np.float32)
    assert lib.mm_init_into(ffi.NULL, 4) == ffi.NULL
    assert lib.mm_init_into(ffi.cast("float*", x.ctypes.data), 0) == ffi.NULL
    assert lib.mm_init_into(ffi.cast("float*", x.ctypes.data), -1) == ffi.NULL
