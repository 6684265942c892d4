"""The bench's roofline names a recorded DRAM traffic for the kernel it runs."""

import os

import bench


def test_the_default_frame_kernel_has_a_traffic_record():
    """Bytes per launch of the headline workload (256 clips of 30 s): at least
    the input once and most of the log-mel rows (the rest may still be in L2
    when the kernel ends), and no second pass over the input."""
    frames = 256 * (1 + 661500 // 512)
    samples, rows = 4 * 256 * 661500, 4 * 128 * frames
    got = bench.recorded_traffic(bench.frame_kernel_name(3))
    assert got is not None
    assert samples <= got <= 1.1 * (samples + rows)
    assert bench.recorded_traffic("no_such_kernel<11>") is None


def test_profiles_name_kernels_that_exist():
    root = os.path.dirname(os.path.abspath(bench.__file__))
    sources = ""
    for f in os.listdir(os.path.join(root, "metalmom_b200", "csrc")):
        sources += open(os.path.join(root, "metalmom_b200", "csrc", f)).read()
    for f in os.listdir(os.path.join(root, "profiles")):
        kernel = f.split("_kernel_")[0] + "_kernel" if "_kernel_" in f else None
        assert kernel is None or kernel in sources, f
