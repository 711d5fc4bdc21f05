"""NVFP4 quantiser around the longest row that it copies to shared memory
(1024 samples), odd lengths, 8-byte aligned input, and the untuned choice
between the two correlator kernels, against the restated quantiser."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import oracle  # noqa: E402

from ftd_b200 import Correlator, tri_size  # noqa: E402
from ftd_b200._lib import COMPUTE_FP4, COMPUTE_FP4_SPLIT, IN_FP32, OUT_FP32  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("K", [7, 9, 127, 1000, 1023, 1024, 1025])
def test_matches_restated_quantiser(K, offset):
    B, N = 2, 70
    v = oracle.workload4_voltages(500 + K, B, N, K)  # RFI bursts: permuted time order
    flat = np.concatenate([np.zeros(offset, np.complex64), v.reshape(-1)])
    A = torch.from_numpy(flat.view(np.float32)).to(DEV)[2 * offset:]
    i, j = np.tril_indices(N)
    order = np.lexsort((j, i))
    diag = i[order] == j[order]
    with Correlator() as c:
        for compute, split, tol in ((COMPUTE_FP4, False, 1e-6), (COMPUTE_FP4_SPLIT, True, 1e-5)):
            C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
            c.herk(A, C, N, K, B, input=IN_FP32, compute=compute, output=OUT_FP32, tune=False)
            assert c.device_status() == 0
            ref = oracle.herk_nvfp4(v, split)
            err = np.abs(C.double().cpu().numpy() - ref)
            # FP32 accumulation (and, split, a lo code flipped by the residual's last bit)
            assert err[:, ~diag].max() <= tol * np.abs(ref).max()


# a size that takes the pair, and shapes with too few k-blocks, rounds or inputs for it
@pytest.mark.parametrize("N,K,B,pair", [(2048, 1024, 8, 2), (2048, 512, 4, 0), (2048, 128, 4, 0),
                                        (1024, 512, 16, 0)])
def test_untuned_equals_both_kernels(N, K, B, pair):
    g = torch.Generator(device=DEV).manual_seed(5)
    A = torch.randn(B, N, K, 2, device=DEV, generator=g)
    outs = []
    for mode in (None, 0, 2):
        C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
        with Correlator() as c:
            if mode is not None:
                c.set_strategy(mode, 0)
            c.herk(A, C, N, K, B, input=IN_FP32, compute=COMPUTE_FP4, output=OUT_FP32, tune=False)
            assert c.last_strategy()["store_mode"] == (pair if mode is None else mode)
            assert c.device_status() == 0
        outs.append(C)
    scale = float(outs[0].abs().max())
    for o in outs[1:]:  # the same quantised products, FP32 sums in another order
        assert float((o - outs[0]).abs().max()) <= 1e-5 * scale
