"""Kernels that start while the one before them ends read what that one writes
with ordinary loads: the read-only path takes data that no one changes while
the reading kernel runs.  Checked on the source (CPU)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ftd_b200", "csrc")

# kernel -> (file, parameters that the kernel in front of it may write)
READS = {
    "quantize_kernel": ("precision.cu", ["amax_bits"]),
    "nvfp4_order_kernel": ("herk_fp4.cu", ["flags"]),
    "nvfp4_quant_kernel": ("herk_fp4.cu", ["src", "nflag", "chans", "rscale"]),
    "split_reduce_kernel": ("herk_fp8.cu", ["ws", "chan_scale"]),
    "negate_plane_kernel": ("herk_fp8.cu", []),
}


def definition(name, path):
    txt = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
    m = re.search(r"\b%s\(([^{;]*)\)\s*\{" % name, txt)
    end = txt.index("\n}\n", m.end())
    return m.group(1), txt[m.end():end]


@pytest.mark.parametrize("name", sorted(READS))
def test_ordinary_loads_behind_the_wait(name):
    path, params = READS[name]
    args, body = definition(name, path)
    assert body.index("griddep_wait()") < min([body.index(p) for p in params], default=len(body))
    for p in params:
        assert not re.search(r"__restrict__\s+%s\b" % p, args), p
        assert not re.search(r"__ldg\([^;]*\b%s\b" % p, body), p
    assert not re.search(r"__ldg\([^;]*\bsc\b", body)  # nvfp4_quant_kernel's view of src


def test_every_early_kernel_waits():
    for path in ("adjoint.cu", "herk_fp4.cu", "herk_fp8.cu", "precision.cu"):
        txt = open(os.path.join(CSRC, path)).read()
        for k in re.findall(r"launch_after\(\s*[^,]*,\s*(\w+_kernel)", txt):
            assert "griddep_wait()" in definition(k, path)[1], k
