"""Large results of the one-clip calls are the library's page-locked blocks,
reused once their array is gone: held results must keep their values however
many calls follow (past the pool's 64 MB they are malloc'd), from several
threads, and for views and in-place changes; results released through the C
ABI go back the same way."""

import gc
import os
import threading

import numpy as np
import pytest

import metalmom_b200 as M
from metalmom_b200._bridge import OWN_BYTES, take_buffer
from metalmom_b200._native import ffi, lib

pytestmark = pytest.mark.gpu


def _clip(seed, n=300000):
    return (0.3 * np.random.default_rng(seed).standard_normal(n)).astype(np.float32)


def test_held_results_keep_their_values():
    first = [M.stft(_clip(i)) for i in range(40)]  # 40 x 2.4 MB
    assert first[0].nbytes >= OWN_BYTES and first[0].flags.writeable
    copies = [a.copy() for a in first]
    rows = [a[3:7] for a in first]  # views outlive their array
    del first
    gc.collect()
    again = [M.stft(_clip(i)) for i in range(40)]
    for i in range(40):
        np.testing.assert_array_equal(again[i], copies[i])
        np.testing.assert_array_equal(rows[i], copies[i][3:7])
    again[0][:] = -1.0
    np.testing.assert_array_equal(M.stft(_clip(0)), copies[0])
    np.testing.assert_array_equal(again[1], copies[1])


def test_sizes_around_the_thresholds_and_several_threads():
    want = {n: M.melspectrogram(_clip(n, n)).copy() for n in (200000, 262143, 262144, 270000, 900001)}
    bad = []

    def work(n):
        for _ in range(15):
            got = M.melspectrogram(_clip(n, n))
            if not np.array_equal(got, want[n]):
                bad.append(n)

    ts = [threading.Thread(target=work, args=(n,)) for n in want for _ in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    x = np.abs(_clip(5, 1 << 19)) + 1e-3
    np.testing.assert_allclose(M.power_to_db(x, top_db=None), 10 * np.log10(x.astype(np.float64)), atol=1e-3)


def test_c_abi_contexts_of_both_kinds_give_the_same_values():
    y = _clip(9)
    p = ffi.new("MMSTFTParams*")
    p.n_fft, p.hop_length, p.win_length, p.center = 2048, 512, 2048, 1
    got = []
    for init in (lib.mm_init, lib.mm_init_pooled, lib.mm_init):
        ctx = init()
        out = ffi.new("MMBuffer*")
        assert lib.mm_stft(ctx, ffi.cast("const float*", y.ctypes.data), len(y), 22050, p, out) == 0
        lib.mm_destroy(ctx)
        n = int(out.count)
        got.append(np.frombuffer(ffi.buffer(out.data, 4 * n), dtype=np.float32).copy())
        lib.mm_buffer_free(out)
        assert out.data == ffi.NULL
        lib.mm_buffer_free(out)
    np.testing.assert_array_equal(got[0], got[1])
    np.testing.assert_array_equal(got[0], got[2])
    out = ffi.new("MMBuffer*")
    ctx = lib.mm_init_pooled()
    assert lib.mm_stft(ctx, ffi.cast("const float*", y.ctypes.data), len(y), 22050, p, out) == 0
    lib.mm_destroy(ctx)
    a = take_buffer(out)
    assert out.data == ffi.NULL
    np.testing.assert_array_equal(a.ravel(), got[0])


def test_a_forked_child_has_its_own_copy():
    """As with any array: a child reads what was there, its writes stay with it,
    and the block goes on receiving results in the parent."""
    y = _clip(11)
    a = M.stft(y)
    want = a.copy()
    pid = os.fork()
    if pid == 0:  # no CUDA here
        same = np.array_equal(a, want)
        a[:] = -1.0
        os._exit(0 if same else 3)
    assert os.waitpid(pid, 0)[1] == 0
    np.testing.assert_array_equal(a, want)
    del a
    gc.collect()
    for _ in range(3):
        np.testing.assert_array_equal(M.stft(y), want)
