"""Corner turn at the alignments its loads distinguish (slices that start on 16
bytes, on 4, on any), at the edges of its 128 x 128 tiles, and for the
XEngine's payload strides.  Integer voltages: bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import oracle  # noqa: E402

from ftd_b200 import Correlator, tri_size  # noqa: E402
from ftd_b200._lib import LAYOUT_TIME_ANT_CHAN_POL  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def on_device(raw, offset):
    buf = torch.zeros(raw.size + offset, dtype=torch.uint8, device=DEV)
    buf[offset:] = torch.from_numpy(np.ascontiguousarray(raw).reshape(-1))
    return buf[offset:]


# ant * chan * pol: 16, 128, 144 (16-byte slices), 132, 20 (4-byte), 130, 77 (any)
@pytest.mark.parametrize("a,c,p", [(8, 1, 2), (32, 2, 2), (36, 2, 2), (33, 2, 2), (5, 2, 2),
                                   (65, 1, 2), (11, 7, 1)])
@pytest.mark.parametrize("K", [1, 4, 127, 128, 131])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_tacp(a, c, p, K, offset):
    ti = 2
    raw = np.random.default_rng(a + K).integers(0, 256, size=ti * K * a * c * p, dtype=np.uint8)
    bf = oracle.ftd_to_batch_first(raw, a, c, p, ti * K, ti, LAYOUT_TIME_ANT_CHAN_POL, False)
    ref = oracle.herk_qc(bf, a, bf.shape[2], bf.shape[0]).astype(np.float32)
    C = torch.full((c * p * ti, tri_size(a), 2), float("nan"), device=DEV)
    with Correlator() as h:
        h.herk_ftd(on_device(raw, offset), C, a, c, p, ti * K, ti)
        assert h.device_status() == 0
    assert np.array_equal(C.cpu().numpy(), ref)


@pytest.mark.parametrize("n", [16, 48, 52, 50, 129, 144])
@pytest.mark.parametrize("offset", [0, 4])
def test_xengine_payload(n, offset):
    K, B = 130, 3
    raw = np.random.default_rng(n).integers(0, 256, size=(B, K, n), dtype=np.uint8)
    out = torch.full((B, tri_size(n), 2), float("nan"), device=DEV)
    with Correlator() as h:
        h.xengine(on_device(raw, offset), out, n, K, B, mat_format=1)
        assert h.device_status() == 0
    got = out.double().cpu().numpy()
    assert np.array_equal(got[..., 0] + 1j * got[..., 1], oracle.xengine(raw, n, K, B, 1))
