"""Calls of many kinds queued on one stream of one handle without a
synchronisation between them.  They share the operand planes, the split-K
partials and the scale buffer, and dependent kernels start early, so a missing
wait or an overwrite shows as a difference from the same calls made one by one
on a handle of their own.  Inputs and outputs differ from round to round.  Every
result is compared bit for bit (each kernel sums in a fixed order)."""
import pytest

torch = pytest.importorskip("torch")

from ftd_b200 import Correlator, tri_size  # noqa: E402
from ftd_b200._lib import (COMPUTE_FP4, COMPUTE_FP4_SPLIT, COMPUTE_FP8, COMPUTE_FP8_SPLIT,  # noqa: E402
                           IN_FP16, IN_FP32, IN_INT4, OUT_FP16, OUT_FP32)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def qc(g, *shape):
    return torch.randint(0, 256, shape, device=DEV, dtype=torch.uint8, generator=g)


def floats(g, b, n, k):
    v = torch.randn(b, n, k, 2, device=DEV, generator=g)
    v[:, : max(1, n // 20), : max(1, k // 100)] *= 20
    return v


def vis(b, n, dt=torch.float32):
    return torch.full((b, tri_size(n), 2), float("nan"), device=DEV, dtype=dt)


def int4(n, k, b, off=0, out=OUT_FP32):
    def make(g):
        A = qc(g, b * n * k + off)[off:]
        C = vis(b, n, torch.float32 if out == OUT_FP32 else torch.float16)
        return C, lambda c: c.herk(A, C, n, k, b, input=IN_INT4, output=out, tune=False)
    return make


def real(n, k, b, compute):
    def make(g):
        A, C = floats(g, b, n, k), vis(b, n)
        return C, lambda c: c.herk(A, C, n, k, b, input=IN_FP32, compute=compute, output=OUT_FP32,
                                   tune=False)
    return make


def half(n, k, b):
    def make(g):
        A, C = floats(g, b, n, k).to(torch.float16), vis(b, n, torch.float16)
        return C, lambda c: c.herk(A, C, n, k, b, input=IN_FP16, output=OUT_FP16, tune=False)
    return make


def kahan(n, k, b):
    def make(g):
        A, S, comp = qc(g, b, n, k), torch.zeros_like(vis(b, n)), torch.zeros_like(vis(b, n))
        return S, lambda c: c.herk_kahan(A, S, comp, n, k, b, input=IN_INT4)
    return make


def raw(a, ch, p, k):
    def make(g):
        R, C = qc(g, k * a * ch * p), vis(ch * p, a)
        return C, lambda c: c.herk_ftd(R, C, a, ch, p, k)
    return make


def payload(n, k, b):
    def make(g):
        P, C = qc(g, b, k, n), vis(b, n)
        return C, lambda c: c.xengine(P, C, n, k, b, mat_format=1)
    return make


def uneven(rows):
    def make(g):
        chans = [{"A": qc(g, rows, 64 * k), "n_inputs": rows - 5 * k, "K": 64 * k,
                  "C": vis(1, rows - 5 * k)[0]} for k in (2, 5, 3)]
        return [ch["C"] for ch in chans], lambda c: c.herk_batched_v(chans)
    return make


def adjoint(n, k, b):
    def make(g):
        G = torch.randn(b, n, n, 2, device=DEV, generator=g)
        V, dV = qc(g, b, n, k), torch.full((b, n, k, 2), float("nan"), device=DEV)
        return dV, lambda c: c.herk_adjoint(G, V, dV, n, k, b, input=IN_INT4)
    return make


# fused, apart, split either way, FP16 out; float promotion in one cooperative and in
# two kernels, hi + lo, NVFP4 on both kernels; the entry points that share the buffers
KINDS = [int4(128, 256, 32), int4(64, 8192, 1), int4(64, 8191, 1), int4(702, 500, 4, out=OUT_FP16),
         real(300, 257, 3, COMPUTE_FP8), real(300, 1000, 1, COMPUTE_FP8), int4(256, 2048, 4, off=3),
         real(200, 4096, 2, COMPUTE_FP8_SPLIT), half(260, 500, 3), real(70, 999, 2, COMPUTE_FP4),
         kahan(130, 512, 2), real(2048, 1024, 8, COMPUTE_FP4), adjoint(136, 100, 3), raw(100, 2, 2, 300),
         real(300, 1030, 2, COMPUTE_FP4_SPLIT), payload(150, 400, 3),
         real(3100, 1010, 2, COMPUTE_FP8), int4(512, 4096, 1), adjoint(264, 257, 1)]


# a new set of uneven channels uploads its descriptors, which waits: last in a round
LAST = [uneven(300)]


def flat(out):
    return out if isinstance(out, list) else [out]


def test_queued_calls_equal_single_calls():
    orders = []
    for r in range(3):  # each round in another order
        step = (1, 3, 7)[r]
        orders.append([KINDS[(i * step) % len(KINDS)] for i in range(len(KINDS))] + LAST)
    with Correlator() as shared:
        for make in KINDS + LAST:  # the buffers reach their sizes: no call below waits for one to grow
            make(torch.Generator(device=DEV).manual_seed(0))[1](shared)
        torch.cuda.synchronize()
        queued = []
        for r, order in enumerate(orders):
            calls = [make(torch.Generator(device=DEV).manual_seed(100 * r + i))
                     for i, make in enumerate(order)]
            torch.cuda.synchronize()
            for _, call in calls:
                call(shared)
            queued.append(calls)
        assert shared.device_status() == 0
        for r, order in enumerate(orders):
            for i, make in enumerate(order):
                out, call = make(torch.Generator(device=DEV).manual_seed(100 * r + i))
                with Correlator() as alone:
                    call(alone)
                    torch.cuda.synchronize()
                    assert alone.device_status() == 0
                for x, y in zip(flat(out), flat(queued[r][i][0])):
                    assert bool(torch.isfinite(x).all()) or x.dtype == torch.float16
                    assert torch.equal(x.view(torch.uint8), y.view(torch.uint8)), (r, i)
