"""The untuned rule and the split-K partial buffer, on the CPU: the buffer that
a caller's graph was captured with outlives its replacement, a failed allocation
leaves the unsplit kernel, init_herk's size covers every shape up to the one it was
given, and the blocks of a promotion pass are resident at once."""
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("strategy") / "strategy_check")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "strategy_check.cpp"),
                    "-I", os.path.join(ROOT, "ftd_b200", "csrc")], check=True, capture_output=True)

    def run(lines):
        r = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
        return [tuple(int(x) for x in ln.split()) for ln in r.stdout.splitlines()]
    return run


def test_partial_buffer_fallback_and_promotion_blocks(check):
    assert check([]) == []


def test_a_smaller_shape_can_need_more(check):
    (_, s4, b4), (_, s2, b2) = check(["rule 148 512 8192 4 1 1", "rule 148 512 8192 2 1 1"])
    assert s2 > s4 > 1 and b2 > b4


def test_bound_covers_every_smaller_shape(check):
    rng = random.Random(3)
    lines, caps = [], []
    for _ in range(400):
        n, k, b = rng.randint(1, 4096), int(2 ** rng.uniform(0, 17)), rng.randint(1, 64)
        lines.append(f"bound {n} {k} {b}")
        for _ in range(20):
            lines.append(f"rule 148 {rng.randint(1, n)} {rng.randint(1, k)} {rng.randint(1, b)} "
                         f"{rng.randint(0, 1)} 1")
    out = check(lines)
    split = 0
    for i in range(0, len(out), 21):
        caps = [o[2] for o in out[i + 1:i + 21]]
        split += sum(c > 0 for c in caps)
        assert max(caps) <= out[i][0]
    assert split > 500


# pairs, inputs, k-blocks, channels, hi + lo: what was measured slower on the CTA
# pair stays on the single CTA, what was faster takes the pair
@pytest.mark.parametrize("args,mode", [
    ((74, 1024, 4, 16, 0), 0), ((74, 1024, 4, 16, 1), 0), ((74, 1024, 16, 52, 1), 0),
    ((74, 512, 8, 65, 1), 0), ((74, 300, 8, 97, 0), 0), ((74, 2048, 4, 5, 0), 0),
    ((74, 2048, 3, 14, 0), 0), ((74, 1500, 16, 3, 1), 0), ((0, 4096, 8, 16, 0), 0),
    ((74, 1100, 8, 19, 1), 2), ((74, 2048, 4, 4, 1), 2), ((74, 2048, 8, 8, 0), 2),
    ((74, 4096, 8, 16, 0), 2), ((74, 4096, 4, 4, 0), 2)])
def test_nvfp4_kernel(check, args, mode):
    assert check(["fp4 " + " ".join(str(a) for a in args)]) == [(mode,)]
