"""Calling the C ABI from Python: one context per call, the library-owned
output buffer handed over as a NumPy array, and a RuntimeError naming the
entry point and its status on failure (the error behaviour of MetalMom's
Python wrappers, which build a context per call as well)."""

import math

import numpy as np

from ._native import ffi, lib

# From this size on the array is the library's buffer itself, released with the
# array; below it a copy costs less than keeping track (30 s of audio: the
# magnitude STFT is 5.3 MB, whose two host copies took 0.6 of its 0.96 ms).
OWN_BYTES = 256 << 10


class _Result:
    """A library-owned buffer that an array keeps alive."""

    def __init__(self, buf, shape):
        own = ffi.new("MMBuffer*")
        own[0] = buf[0]
        buf.data = ffi.NULL  # moved
        self.buf = ffi.gc(own, lib.mm_buffer_free)
        self.__array_interface__ = {"shape": shape, "typestr": "<f4", "version": 3,
                                    "data": (int(ffi.cast("uintptr_t", own.data)), False)}


def take_buffer(buf):
    """The floats of a filled MMBuffer as an array of its shape; the C buffer
    is released at once, or with the array when it is large (an empty result
    has data NULL and count 0 with the shape set)."""
    try:
        shape = tuple(int(buf.shape[d]) for d in range(buf.ndim))
        n = int(buf.count)
        if n == 0 or buf.data == ffi.NULL:
            return np.empty(shape, dtype=np.float32)
        if 4 * n >= OWN_BYTES:
            if math.prod(shape) != n:
                raise ValueError(f"a buffer of {n} floats cannot take the shape {shape}")
            return np.asarray(_Result(buf, shape))
        view = np.frombuffer(ffi.buffer(buf.data, 4 * n), dtype=np.float32)
        return view.reshape(shape).copy()
    finally:
        lib.mm_buffer_free(buf)


def bridge_call(name, fn, *args):
    """fn(ctx, *args, out) inside a fresh context; the output as an array."""
    ctx = lib.mm_init_pooled()
    if ctx == ffi.NULL:
        raise RuntimeError("Failed to initialize MetalMom context")
    try:
        out = ffi.new("MMBuffer*")
        status = fn(ctx, *args, out)
        if status != 0:
            raise RuntimeError(f"{name} failed with status {status}")
        return take_buffer(out)
    finally:
        lib.mm_destroy(ctx)


def float_ptr(a):
    """A contiguous float32 view of `a` and its cffi pointer (keep the view
    alive while the pointer is in use)."""
    a = np.ascontiguousarray(a, dtype=np.float32)
    return a, ffi.cast("const float*", a.ctypes.data)


def stft_params(n_fft, hop, win, center):
    p = ffi.new("MMSTFTParams*")
    p.n_fft, p.hop_length, p.win_length, p.center = n_fft, hop, win, 1 if center else 0
    return p
