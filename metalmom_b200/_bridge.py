"""Calling the C ABI from Python: one context per call, the output as a NumPy
array, and a RuntimeError naming the entry point and its status on failure (the
error behaviour of MetalMom's Python wrappers, which build a context per call
as well).

Every result is an ordinary array: its memory is NumPy's own and pageable, so
that nothing reuses it while the caller, or an asynchronous copy that the
caller has queued, still reads it."""

import math

import numpy as np

from ._native import ffi, lib
from .shard import frames_of

# From this size on the array is made before the call and the library copies
# the result into it, piece by piece while the rest crosses the bus; below it
# the library's own buffer is copied afterwards.  30 s of audio, host to host:
# magnitude STFT (5.3 MB) 988 us with both copies, 552-598 us so; mel
# spectrogram (0.66 MB) 297 and 247-276 us.
OWN_BYTES = 256 << 10


def take_buffer(buf):
    """The floats of a filled MMBuffer as a new array of its shape; the C
    buffer is released whatever happens (an empty result has data NULL and
    count 0 with the shape set)."""
    try:
        shape = tuple(int(buf.shape[d]) for d in range(buf.ndim))
        n = int(buf.count)
        if n == 0 or buf.data == ffi.NULL:
            return np.empty(shape, dtype=np.float32)
        view = np.frombuffer(ffi.buffer(buf.data, 4 * n), dtype=np.float32)
        return view.reshape(shape).copy()
    finally:
        lib.mm_buffer_free(buf)


def frame_shape(rows, length, n_fft, hop, center, *rest):
    """(rows, frames, *rest) of a call's result, None where the call decides."""
    try:
        n_fft, hop = int(n_fft), int(hop)
    except (TypeError, ValueError, OverflowError):
        return None
    if n_fft <= 0 or hop <= 0:
        return None
    return (rows, frames_of(length, n_fft, hop, center), *rest)


def sample_shape(n_frames, n_fft, hop, center, length):
    """(samples,) of an inverse transform's result, as ``frame_shape``."""
    try:
        hop, length = int(hop), int(length)
    except (TypeError, ValueError, OverflowError):
        return None
    return (length if length > 0 else (n_frames - 1) * hop + (0 if center else n_fft),)


def _empty(shape):
    """An array for a large result of that shape, else None."""
    try:
        if shape is None or min(shape) <= 0 or 4 * math.prod(shape) < OWN_BYTES:
            return None
        return np.empty(shape, dtype=np.float32)
    except (MemoryError, TypeError, ValueError):  # the call itself says what is wrong with its arguments
        return None


def bridge_call(name, fn, *args, shape=None):
    """fn(ctx, *args, out) inside a fresh context; the output as an array.
    ``shape``: that of the result as far as it is known; a result of another
    size or shape is returned all the same, only less directly."""
    dst = _empty(shape)
    into = ffi.NULL if dst is None else ffi.cast("float*", dst.ctypes.data)
    ctx = lib.mm_init() if dst is None else lib.mm_init_into(into, dst.size)
    if ctx == ffi.NULL:
        raise RuntimeError("Failed to initialize MetalMom context")
    try:
        out = ffi.new("MMBuffer*")
        status = fn(ctx, *args, out)
        if status != 0:
            raise RuntimeError(f"{name} failed with status {status}")
        if dst is None or out.data != into:
            return take_buffer(out)
        got = tuple(int(out.shape[d]) for d in range(out.ndim))
        return dst if got == dst.shape else dst.reshape(got)
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
