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
