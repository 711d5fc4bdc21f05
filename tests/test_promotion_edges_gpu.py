"""Promotion passes at the sizes where they can go wrong: rows that are no
multiple of 16 or 4 samples, inputs that start on any byte, fewer rows than a
block holds, and one chunk per row.  Integer voltages are exact, so every
comparison is bit for bit against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import oracle  # noqa: E402

from ftd_b200 import Correlator, tri_size  # noqa: E402
from ftd_b200._lib import IN_INT4, OUT_FP32  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def on_device(data, offset):
    """The bytes on the device, starting `offset` bytes past an allocation's start."""
    buf = torch.zeros(data.size + offset, dtype=torch.uint8, device=DEV)
    buf[offset:] = torch.from_numpy(data.reshape(-1))
    return buf[offset:]


# store modes: 0 E4M3 planes, 4 FP6 planes, 10 signed 8-bit planes (CTA pair)
@pytest.mark.parametrize("mode", [0, 4, 10])
@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("K", [1, 2, 3, 5, 15, 17, 31, 130, 500, 511])
def test_ragged_rows_and_offsets(K, offset, mode):
    N, B = 37, 3
    qc = oracle.gaussian_qc(K + offset, B, N, K)
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    with Correlator() as c:
        c.set_strategy(mode, 0)
        c.herk(on_device(qc, offset), C, N, K, B, input=IN_INT4, output=OUT_FP32, tune=False)
        assert c.device_status() == 0
    assert np.array_equal(C.cpu().numpy(), oracle.herk_qc(qc, N, K, B).astype(np.float32))


@pytest.mark.parametrize("K,lda,offset", [(1, 1, 1), (77, 77, 2), (64, 67, 3), (500, 500, 4),
                                          (130, 144, 0)])
def test_gathered_rows(K, lda, offset):
    rows, n = 40, 33
    block = oracle.gaussian_qc(K, 1, rows, lda)[0]
    active = np.sort(np.random.default_rng(K).choice(rows, size=n, replace=False)).astype(np.int32)
    ch = {"A": on_device(block, offset), "C": torch.full((tri_size(n), 2), float("nan"), device=DEV),
          "n_inputs": n, "K": K, "lda": lda, "active": torch.from_numpy(active).to(DEV)}
    with Correlator() as c:
        c.herk_batched_v([ch])
        assert c.device_status() == 0
    qc = np.ascontiguousarray(block[active][:, :K]).reshape(1, n, K)
    assert np.array_equal(ch["C"].cpu().numpy(), oracle.herk_qc(qc, n, K, 1)[0].astype(np.float32))


# rows per block: the least (one piece per thread), between, and the most
@pytest.mark.parametrize("N,K,B", [(3, 16, 1), (700, 256, 24), (512, 2048, 40)])
def test_block_sizes(N, K, B):
    qc = oracle.gaussian_qc(N, B, N, K)
    C = torch.full((B, tri_size(N), 2), float("nan"), device=DEV)
    with Correlator() as c:
        c.set_strategy(0, 0)
        c.herk(torch.from_numpy(qc.reshape(-1)).to(DEV), C, N, K, B, input=IN_INT4,
               output=OUT_FP32, tune=False)
        assert c.device_status() == 0
    rows = oracle.herk_qc_rows(qc, N, K, B - 1, max(0, N - 8), N).astype(np.float32)
    got = C[B - 1, tri_size(max(0, N - 8)):].cpu().numpy()
    assert np.array_equal(got, rows)
    assert np.array_equal(C[0, :10].cpu().numpy(),
                          oracle.herk_qc_rows(qc, N, K, 0, 0, min(N, 4)).astype(np.float32)[:10])
