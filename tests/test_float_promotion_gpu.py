"""Float promotion to scaled E4M3 on both of its paths: channels long enough for
the cooperative kernel and channels below that, one channel and several, the
plain and the split mode, ragged rows.  A channel's largest component lies in
its first rows, so that the restated quantiser of those rows alone gives the
expected triangle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import oracle  # noqa: E402

from ftd_b200 import Correlator, tri_size  # noqa: E402
from ftd_b200._lib import COMPUTE_FP8, COMPUTE_FP8_SPLIT, IN_FP32, OUT_FP32  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# 25 MB a channel (cooperative), one short channel (cooperative), short ones
@pytest.mark.parametrize("N,K,B", [(3100, 1010, 3), (3100, 1009, 2), (33, 7, 1), (300, 257, 1),
                                   (33, 7, 5), (300, 257, 7), (700, 1000, 3)])
def test_first_rows_match_the_restated_quantiser(N, K, B):
    g = torch.Generator(device=DEV).manual_seed(N + K)
    A = torch.randn(B, N, K, 2, device=DEV, generator=g)
    A *= torch.tensor([0.01, 1.0, 30.0, 0.2, 5.0, 1e3, 1e-3], device=DEV)[:B].view(B, 1, 1, 1)
    A[:, 3, K // 2, 1] = 40 * A.abs().amax(dim=(1, 2, 3))
    rows = min(N, 33)
    head = A[:, :rows].cpu().numpy()
    v = np.ascontiguousarray(head[..., 0] + 1j * head[..., 1]).astype(np.complex64)
    with Correlator() as c:
        for compute, split in ((COMPUTE_FP8, False), (COMPUTE_FP8_SPLIT, True)):
            # every 32 samples two products are added to an FP32 sum that drops
            # what lies below its last bit (2^-24 on average): at most K / 16 + 2 times per
            # product of parts, of which the split mode has three (the measured
            # error is about half of this)
            tol = (3 if split else 1) * (K / 16 + 2) * 2.0 ** -24
            C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
            c.herk(A, C, N, K, B, input=IN_FP32, compute=compute, output=OUT_FP32, tune=False)
            assert c.device_status() == 0
            got = C[:, :tri_size(rows)].double().cpu().numpy()
            ref = oracle.herk_fp8_scaled(v, split)
            for b in range(B):
                assert np.abs(got[b] - ref[b]).max() <= tol * np.abs(ref[b]).max()
            assert bool(torch.isfinite(C).all())


# more channels than a grid has rows, on the path of short channels
@pytest.mark.parametrize("compute,split", [(COMPUTE_FP8, False), (COMPUTE_FP8_SPLIT, True)])
def test_more_than_65535_channels(compute, split):
    N, K, B = 2, 16, 65537
    g = torch.Generator(device=DEV).manual_seed(7)
    A = torch.randn(B, N, K, 2, device=DEV, generator=g)
    A *= torch.exp(4 * torch.randn(B, 1, 1, 1, device=DEV, generator=g))
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    with Correlator() as c:
        c.herk(A, C, N, K, B, input=IN_FP32, compute=compute, output=OUT_FP32, tune=False)
        assert c.device_status() == 0
    got = C.double().cpu().numpy()
    v = np.ascontiguousarray(A.cpu().numpy()).view(np.complex64)[..., 0]
    for b in (0, 1, 65534, 65535, 65536):
        tol = (3 if split else 1) * (K / 16 + 2) * 2.0 ** -24  # as above
        ref = oracle.herk_fp8_scaled(v[b:b + 1], split)[0]
        assert np.abs(got[b] - ref).max() <= tol * np.abs(ref).max()
    # every channel: E4M3 rounds each part by at most 2^-4 of it, so a product of
    # two by 2^-3 + 2^-8, and what is below its normal range by 2^-10 of 1 / scale
    w = v.astype(np.complex128)
    i, j = np.array([0, 1, 1]), np.array([0, 0, 1])
    bound = 0.13 * (np.abs(w[:, i]) * np.abs(w[:, j])).sum(-1)
    bound += 1e-4 * np.abs(w).max(axis=(1, 2))[:, None] ** 2
    exact = (w[:, i] * np.conj(w[:, j])).sum(-1)
    assert (np.abs(got[..., 0] + 1j * got[..., 1] - exact) <= bound).all()
