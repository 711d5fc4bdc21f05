"""Adjoint and gain gradient at the edges of their tiles: fewer antennas and
samples than one tile, one more than a whole number, odd sample counts, and
several channels; each against FP64 with a bound that follows from the
arithmetic."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import oracle  # noqa: E402

from ftd_b200 import Correlator, tri_size  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N,K,B", [(8, 1, 1), (8, 17, 5), (24, 64, 2), (64, 63, 3), (128, 128, 1),
                                   (136, 65, 2), (200, 130, 3), (264, 257, 2), (520, 40, 1)])
@pytest.mark.parametrize("offset", [0, 1])
def test_adjoint_edges(N, K, B, offset):
    rng = np.random.default_rng(N + K)
    G = (rng.normal(size=(B, N, N)) + 1j * rng.normal(size=(B, N, N))).astype(np.complex64)
    qc = oracle.gaussian_qc(N * K, B, N, K)
    dG = torch.from_numpy(G.view(np.float32)).to(DEV)
    buf = torch.zeros(qc.size + offset, dtype=torch.uint8, device=DEV)
    buf[offset:] = torch.from_numpy(qc.reshape(-1))
    out = torch.full((B, N, K, 2), float("nan"), device=DEV)
    with Correlator() as c:
        for _ in range(2):  # the second call finds the first one's workspace
            c.herk_adjoint(dG, buf[offset:], out, N, K, B)
        assert c.device_status() == 0
    o = out.double().cpu().numpy()
    re, im = oracle.decode_qc(qc)
    V = re.astype(np.float64) + 1j * im
    S = G.astype(np.complex128) + np.conj(np.transpose(G.astype(np.complex128), (0, 2, 1)))
    # S = hi + lo in bf16 leaves 2^-17 of each part (twice, and FP32's own
    # rounding of the sum, in the bound); FP32 sums of 4 N products add N 2^-22
    bound = (2.0 ** -15 + N * 2.0 ** -22) * (np.abs(S) @ np.abs(V)) + 1e-30
    assert (np.abs(o[..., 0] + 1j * o[..., 1] - S @ V) <= bound).all()


@pytest.mark.parametrize("N,B", [(1, 1), (2, 3), (31, 2), (63, 1), (64, 2), (65, 2), (127, 1),
                                 (128, 2), (129, 3), (193, 1), (300, 2)])
def test_gain_gradient_edges(N, B):
    rng = np.random.default_rng(N)
    P = tri_size(N)

    def vis():
        v = rng.normal(size=(B, P, 2)).astype(np.float32)
        v[:, [i * (i + 1) // 2 + i for i in range(N)], 1] = 0
        return v
    Ro, Rm = vis(), vis()
    W = rng.uniform(size=(B, P)).astype(np.float32)
    g = (rng.normal(size=N) + 1j * rng.normal(size=N)).astype(np.complex64)
    L_ref, grad_ref = oracle.gain_loss_grad(Ro, Rm, W, g.astype(np.complex128), N)
    grad = torch.full((N, 2), float("nan"), dtype=torch.float64, device=DEV)
    loss = torch.full((1,), float("nan"), dtype=torch.float64, device=DEV)
    dev = [torch.from_numpy(x).to(DEV) for x in (Ro, Rm, W)]
    gd = torch.from_numpy(np.stack([g.real, g.imag], -1)).to(DEV)
    with Correlator() as c:
        c.gain_gradient(*dev, gd, N, B, grad, loss)
    torch.cuda.synchronize()
    got = grad[:, 0].cpu().numpy() + 1j * grad[:, 1].cpu().numpy()
    # FP32 terms and sums of at most 128 terms in a tile, FP64 across tiles
    assert abs(float(loss.item()) - L_ref) <= 1e-5 * L_ref
    assert np.abs(got - grad_ref).max() <= 2e-5 * np.abs(grad_ref).max()
