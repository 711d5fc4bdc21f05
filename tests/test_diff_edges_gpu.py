"""Gain gradient and adjoint at the edges of their tiles, each against FP64
with a bound that follows from the arithmetic."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import oracle  # noqa: E402

from ftd_b200 import Correlator, tri_size  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


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
