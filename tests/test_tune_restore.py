"""Reading the launch choice, setting another and setting back what was read
leaves the library's own choice as it was, and the choice that is reported is
the one that runs.  In a process of its own: the choice is process-wide."""

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import metalmom_b200 as M
from metalmom_b200._native import lib
own = {1 << b: 3 if 8 <= b <= 12 else 0 for b in range(4, 16)}
def runs():
    return {n: lib.mm_tune_get(n) for n in own}
def python_runs():
    return {n: M.tune_variant(n) for n in own}
assert runs() == own == python_runs(), runs()
for n in own:  # the C functions
    old = lib.mm_tune_get(n)
    for v in (0, 1, 2, 3):
        assert lib.mm_tune_set(n, v) == 0 and lib.mm_tune_get(n) == v
    assert lib.mm_tune_set(n, old) == 0
assert runs() == own
for n in own:  # the Python functions, and nested
    old = M.tune_get(n)
    for v in (0, 1, 2, 3):
        M.tune_set(n, v)
        assert M.tune_get(n) == M.tune_variant(n) == v
        inner = M.tune_get(n)
        M.tune_set(n, 2)
        M.tune_set(n, inner)
        assert M.tune_get(n) == M.tune_variant(n) == v
    M.tune_set(n, old)
    assert M.tune_get(n) == old
assert runs() == own == python_runs()
M.tune_set(1024, 0)  # asked for, and so kept
assert M.tune_variant(1024) == 0
M.tune_set(1024, M.tune_get(1024))
assert M.tune_variant(1024) == 0
try:
    M.tune_variant(1000)
except RuntimeError as e:
    print(e)
else:
    raise AssertionError("an n_fft that has no variants")
"""


def test_saving_and_restoring_keeps_the_librarys_choice():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
