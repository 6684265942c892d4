"""Kernels that start while the kernel before them finishes (griddep_wait) read
what that kernel writes by ordinary loads.  __ldg is the non-coherent path,
defined only for memory that nobody writes while the kernel lives, and the
compiler may move it ahead of the wait."""

import os
import re

import numpy as np
import pytest

import metalmom_b200 as M
from oracle import oracle as O

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "metalmom_b200", "csrc")

# Tables and descriptors: written before the kernel ahead of them starts.
CONSTANT = {"a.basis", "a.tile_clip", "a.tile_first", "a.clips", "a.window", "a.mel_lane", "a.mel_lw", "a.mel_info",
            "src_words"}


def _functions(text):
    """(name, body) of every function at the outermost level of the file's namespaces."""
    for m in re.finditer(r"^[^\n;{}/]*?(\w+)\([^;{}]*\)\s*\{", text, flags=re.M):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_what_an_early_kernel_reads(name):
    functions = dict(_functions(_source(name)))
    early = [f for f, body in functions.items() if "griddep_wait()" in body]
    # with the functions of the same file that they call
    todo, seen = list(early), set()
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        todo += [g for g in functions if re.search(r"\b%s\b(<[^;()]*>)?\(" % g, functions[f])]
    for f in seen:
        for operand in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?([\w.]+)", functions[f]):
            if name == "frontend_pair.cu" and operand in ("base", "p", "sig", "twq", "a.signal"):
                continue  # samples and twiddles: the kernel ahead only resets the clips' maxima
            assert operand in CONSTANT, f"{name}: {f} reads {operand} through the non-coherent path"
    if name in ("frontend_kernels.cu", "frontend_pair.cu"):
        assert early


@pytest.mark.gpu
@pytest.mark.parametrize("n_mels", [128, 80, 40])  # folded DCT with 128 and 80 bands, pipelined with 40
def test_replays_with_changing_inputs(n_mels):
    """Replays that follow each other without a wait, the input exchanged in
    between on the stream: every replay's rows and maxima are its own.  A clip's
    maximum, 100 dB above most of it, decides the floor and so every value there."""
    import torch
    rng = np.random.default_rng(n_mels)
    n, rounds = 40000, 24
    # most of a clip lies under the floor that its loud end sets
    shape = np.where(np.arange(n) < 0.8 * n, 1e-5, 1.0)
    clips = [(s * shape * rng.standard_normal((3, n))).astype(np.float32) for s in np.geomspace(1e-3, 1.0, rounds)]

    class View:
        def __init__(self, address, count):
            self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (address, False), "version": 2}

    with M.Plan([n] * 3, n_mels=n_mels) as plan:
        src = [torch.as_tensor(View(plan.device_input + 4 * o, n), device="cuda") for o in plan.in_offsets]
        count = max(o + r * f for o, r, f in zip(plan.out_offsets, plan.clip_rows, plan.frames))
        out = torch.as_tensor(View(plan.device_output, count), device="cuda")
        given = [torch.from_numpy(c).cuda() for c in clips]
        got = torch.empty((rounds, count), device="cuda")
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for i in range(rounds):
                for d, g in zip(src, given[i]):
                    d.copy_(g)
                plan.execute(stream=s.cuda_stream)
                got[i].copy_(out)
        s.synchronize()
        got = got.cpu().numpy()
        for i in range(rounds):
            want = M.mfcc_batch(list(clips[i]), n_mels=n_mels)
            for y, w, off in zip(clips[i], want, plan.out_offsets):
                np.testing.assert_array_equal(got[i, off:off + w.size].reshape(w.shape), w)
                exp = O.mfcc(y, 22050, 20, 2048, 512, 2048, n_mels)
                assert O.mfcc_rel_error(w, exp) < 1e-4
