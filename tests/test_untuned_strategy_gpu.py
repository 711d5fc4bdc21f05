"""Untuned calls on a handle that was given no strategy: the kernel (promotion
apart or fused in) and the split of K follow the call's sizes.  Every shape is
bit-exact against the oracle through every entry point that takes the rule, what
was launched is what the rule says, float input split by the rule agrees with
the unsplit kernel, and whatever a call needs under capture is there after
init_herk or after one call of its shape."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import oracle  # noqa: E402

from ftd_b200 import Correlator, tri_size  # noqa: E402
from ftd_b200._lib import (COMPUTE_FP8, COMPUTE_FP8_SPLIT, IN_FP16, IN_FP32, IN_INT4,  # noqa: E402
                           LAYOUT_CHAN_POL_ANT_TIME, LAYOUT_TIME_ANT_CHAN_POL, OUT_FP16, OUT_FP32)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def device_bytes(qc, offset=0):
    buf = torch.zeros(qc.size + offset, dtype=torch.uint8, device=DEV)
    buf[offset:] = torch.from_numpy(qc.reshape(-1))
    return buf[offset:]


def chosen(c):
    st = c.last_strategy()
    return st["store_mode"], st["splits"]


# one tile or several, below and above the splits' reach; K that the fused
# kernel takes (multiples of 16) and that it does not; one k-block.  The last
# two: the ranges of K with the promotion fused in and apart (148 SMs).
@pytest.mark.parametrize("N,K,B,fused,apart", [
    (1, 1, 1, 1, 1), (64, 8192, 1, 22, 16), (64, 8191, 1, 0, 16), (130, 12800, 3, 15, 15),
    (256, 2048, 4, 6, 4), (257, 2050, 4, 0, 5), (128, 256, 32, 1, 1), (300, 128, 60, 1, 1),
    (512, 4096, 1, 8, 8), (40, 30000, 5, 27, 27), (1024, 1024, 16, 0, 1)])
@pytest.mark.parametrize("offset", [0, 3])
def test_bit_exact(N, K, B, fused, apart, offset):
    qc = oracle.gaussian_qc(N + K, B, N, K)
    ref = oracle.herk_qc(qc, N, K, B).astype(np.float32)
    d = device_bytes(qc, offset)
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    C16 = torch.full((B, tri_size(N), 2), float("nan"), device=DEV, dtype=torch.float16)
    S, comp = torch.zeros_like(C), torch.zeros_like(C)
    with Correlator() as c:
        # the fused kernel takes K in multiples of 16 at 16-byte aligned addresses
        want = (16, fused) if K % 16 == 0 and offset == 0 and fused else (0, apart)
        c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
        assert chosen(c) == want
        c.herk(d, C16, N, K, B, input=IN_INT4, output=OUT_FP16, tune=False)
        assert chosen(c) == want
        c.herk_kahan(d, S, comp, N, K, B, input=IN_INT4)
        assert c.last_strategy()["splits"] == 1
        assert c.device_status() == 0
    assert np.array_equal(C.cpu().numpy(), ref)
    # integers beyond half's range: inf on both sides
    with np.errstate(over="ignore"):
        assert np.array_equal(C16.cpu().numpy(), ref.astype(np.float16))
    assert np.array_equal(S.cpu().numpy(), ref)


@pytest.mark.parametrize("layout", [LAYOUT_TIME_ANT_CHAN_POL, LAYOUT_CHAN_POL_ANT_TIME])
@pytest.mark.parametrize("a,ch,p,K", [(100, 1, 2, 4096), (257, 2, 1, 2050), (33, 3, 1, 5000)])
def test_raw_packets_split(layout, a, ch, p, K):
    raw = np.random.default_rng(a).integers(0, 256, size=K * a * ch * p, dtype=np.uint8)
    bf = oracle.ftd_to_batch_first(raw, a, ch, p, K, 1, layout, False)
    C = torch.full((ch * p, tri_size(a), 2), float("nan"), device=DEV)
    with Correlator() as c:
        c.herk_ftd(torch.from_numpy(raw).to(DEV), C, a, ch, p, K, layout=layout)
        assert chosen(c)[0] == 0 and chosen(c)[1] > 1
        assert c.device_status() == 0
    assert np.array_equal(C.cpu().numpy(), oracle.herk_qc(bf, a, K, ch * p).astype(np.float32))


@pytest.mark.parametrize("kind", ["fp16", "fp8", "fp8_split"])
@pytest.mark.parametrize("N,K,B", [(200, 4096, 2), (130, 5000, 3)])
def test_float_input_split_by_the_rule(kind, N, K, B):
    g = torch.Generator(device=DEV).manual_seed(N)
    A = torch.randn(B, N, K, 2, device=DEV, generator=g)
    A *= torch.tensor([0.01, 1.0, 30.0], device=DEV)[:B].view(B, 1, 1, 1)
    kw = {"fp16": dict(input=IN_FP16), "fp8": dict(input=IN_FP32, compute=COMPUTE_FP8),
          "fp8_split": dict(input=IN_FP32, compute=COMPUTE_FP8_SPLIT)}[kind]
    if kind == "fp16":
        A = A.mul_(2.5).to(torch.float16)
    C = [torch.full((B, tri_size(N), 2), float("nan"), device=DEV) for _ in range(2)]
    with Correlator() as c:
        c.herk(A, C[0], N, K, B, output=OUT_FP32, tune=False, **kw)
        assert chosen(c)[1] > 1
        c.set_strategy(0, 0)
        c.herk(A, C[1], N, K, B, output=OUT_FP32, tune=False, **kw)
        assert chosen(c) == (0, 1)
        assert c.device_status() == 0
    # the same products in FP32 sums of another order: per 32 samples and product of
    # parts (three of them for hi + lo) two additions of 2^-24 at most, on either side,
    # and the additions of at most 32 ranges
    tol = 2 * ((3 if kind == "fp8_split" else 1) * (K / 16 + 2) + 32) * 2.0 ** -24
    for b in range(B):
        scale = float(C[1][b].abs().max())
        assert scale > 0 and float((C[0][b] - C[1][b]).abs().max()) <= tol * scale


def test_clear_strategy_is_a_new_handle():
    N, K, B = 64, 8192, 1
    d = device_bytes(oracle.gaussian_qc(5, B, N, K))
    C = torch.empty(B, tri_size(N), 2, device=DEV)
    with Correlator() as c:
        def run():
            c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
            return chosen(c)
        first = run()
        c.set_strategy(2, 0, splits=3)
        assert run() == (2, 3)
        c.clear_strategy()
        assert run() == first == (16, 22)


def test_alpha_beta_on_a_split_call():
    N, K, B = 200, 8192, 2
    qc = oracle.gaussian_qc(9, B, N, K)
    R = oracle.herk_qc(qc, N, K, B)
    old = torch.randn(B, tri_size(N), 2, device=DEV)
    C = old.clone()
    with Correlator() as c:
        c.herk(device_bytes(qc), C, N, K, B, input=IN_INT4, output=OUT_FP32, alpha=0.5, beta=2.0,
               tune=False)
        assert chosen(c) == (16, 16)
        assert c.device_status() == 0
    np.testing.assert_allclose(C.double().cpu().numpy(),
                               0.5 * R + 2.0 * old.double().cpu().numpy(), rtol=1e-6, atol=1e-3)


@pytest.mark.parametrize("prepare", ["init", "call"])
@pytest.mark.parametrize("offset", [0, 3])
def test_capture(prepare, offset):
    # after init_herk, or after one call on an aligned input, the shape can be
    # captured on an input of any alignment, and with Kahan accumulation
    N, K, B = 256, 8192, 2
    qc = oracle.gaussian_qc(11, B, N, K)
    ref = oracle.herk_qc(qc, N, K, B).astype(np.float32)
    d = device_bytes(qc, offset)
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    S, comp = torch.zeros_like(C), torch.zeros_like(C)
    s = torch.cuda.Stream()
    with Correlator() as c:
        if prepare == "init":
            c.init_herk(N, K, B)
        else:
            c.herk(device_bytes(qc), C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
            C.fill_(float("nan"))
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False, stream=s)
            assert chosen(c) == ((0, 13) if offset else (16, 16))
            c.herk_kahan(d, S, comp, N, K, B, input=IN_INT4, stream=s)
        S.zero_(), comp.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(C.cpu().numpy(), ref)
        assert np.array_equal(S.cpu().numpy(), ref)
        assert c.device_status() == 0
        del g


@pytest.mark.parametrize("init", [True, False])
def test_graph_outlives_later_calls(init):
    # a smaller shape takes more partial triangles (seven ranges of 2 channels
    # against three of 4): the caller's graph keeps the buffer it was captured with.
    # None of the later calls needs more operand planes than the captured one.
    N, K, B = 512, 8192, 4
    qc = oracle.gaussian_qc(21, B, N, K)
    d = device_bytes(qc)
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    s = torch.cuda.Stream()
    with Correlator() as c:
        if init:
            c.init_herk(N, K, B)
        else:
            c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False, stream=s)
            assert chosen(c) == (16, 3)
        for n, k, b in ((512, 8192, 2), (256, 32768, 2), (700, 8192, 2)):
            small = oracle.gaussian_qc(n + b, b, n, k)
            out = torch.full((b, tri_size(n), 2), float("nan"), device=DEV)
            c.herk(device_bytes(small), out, n, k, b, input=IN_INT4, output=OUT_FP32, tune=False)
            assert chosen(c)[1] >= 3
            rows = oracle.herk_qc_rows(small, n, k, b - 1, n - 4, n).astype(np.float32)
            assert np.array_equal(out[b - 1, tri_size(n - 4):].cpu().numpy(), rows)
        C.fill_(float("nan"))
        keep = [torch.full((8 << 20,), 7.0, device=DEV) for _ in range(8)]  # what was freed is reused
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(C.cpu().numpy(), oracle.herk_qc(qc, N, K, B).astype(np.float32))
        assert all(bool((t == 7.0).all()) for t in keep)
        assert c.device_status() == 0
        del g


def test_no_memory_for_partials():
    # 33.6 MB of planes fit, 12.6 MB of partial triangles do not: eager and
    # captured calls and the tuner all go on without them
    N, K, B = 512, 8192, 4
    qc = oracle.gaussian_qc(31, B, N, K)
    ref = oracle.herk_qc(qc, N, K, B).astype(np.float32)
    d = device_bytes(qc)
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    s = torch.cuda.Stream()
    with Correlator() as c:  # every kernel is loaded before the memory goes
        c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
        c.tune(d, C, N, K, B)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    with Correlator() as c:
        free = torch.cuda.mem_get_info()[0]
        try:
            hog = torch.empty(free - (40 << 20), dtype=torch.uint8, device=DEV)
        except torch.cuda.OutOfMemoryError:
            pytest.skip("device memory is in use elsewhere")
        try:
            c.init_herk(N, K, B)
            c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
            assert chosen(c)[1] == 1
            assert np.array_equal(C.cpu().numpy(), ref)
            C.fill_(float("nan"))
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False, stream=s)
            assert chosen(c)[1] == 1
            g.replay()
            assert np.array_equal(C.cpu().numpy(), ref)
            del g
            C.fill_(float("nan"))
            c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=True)
            assert np.array_equal(C.cpu().numpy(), ref)
            assert c.tuned_split_k(N, K, B) == 1
            assert c.device_status() == 0
        finally:
            del hog
            torch.cuda.empty_cache()
        c.init_herk(N, K, B)  # tries again
        c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
        assert chosen(c) == (16, 3)


def test_end_herk_gives_the_partials_back():
    N, K, B = 512, 8192, 4
    qc = oracle.gaussian_qc(41, B, N, K)
    d = device_bytes(qc)
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    with Correlator() as c:
        c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)  # kernels loaded
        c.end_herk()
        free = torch.cuda.mem_get_info()[0]
        c.init_herk(N, K, B)
        assert torch.cuda.mem_get_info()[0] <= free - (100 << 20)  # planes and partials
        c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
        c.end_herk()
        assert torch.cuda.mem_get_info()[0] >= free
        c.herk(d, C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
        assert c.device_status() == 0
    assert np.array_equal(C.cpu().numpy(), oracle.herk_qc(qc, N, K, B).astype(np.float32))
