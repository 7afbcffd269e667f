"""The training kernels of the learned guess (marked gpu): the gradient over
batches of odd sizes, one tile to several tiles per CTA, against plain torch
in FP64 (FP32 sums of up to 20,000 terms: 1e-5 of the gradient's norm); two
runs of the same training agree bit for bit (no atomics)."""
import numpy as np
import pytest


def _torch_grad(torch, w, X, T):
    h1 = torch.relu(X @ w[:512].view(64, 8).T + w[512:576])
    h2 = torch.relu(h1 @ w[576:4672].view(64, 64).T + w[4672:4736])
    return ((h2 @ w[4736:4800] + w[4800] - T) ** 2).mean()


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [1, 31, 32, 33, 4097, 9472, 9473, 20001])
def test_gradient_matches_fp64(nb):
    import torch
    from flash5_b200.riemann import ExactRiemann
    g = torch.Generator(device="cuda")
    g.manual_seed(nb)
    X = torch.randn(nb + 5, 8, generator=g, device="cuda")
    T = torch.randn(nb + 5, generator=g, device="cuda")
    idx = torch.randperm(nb + 5, generator=g, device="cuda")[:nb].to(torch.int32)
    rs = ExactRiemann(device=0)
    got, loss = rs.grad(X, T, idx)
    w = torch.from_numpy(rs.weights()).cuda().double().requires_grad_(True)
    ref = _torch_grad(torch, w, X[idx.long()].double(), T[idx.long()].double())
    ref.backward()
    want = float(ref.detach())
    assert abs(loss - want) <= 1e-5 * want
    d = np.linalg.norm(got - w.grad.cpu().numpy())
    assert d <= 1e-5 * float(w.grad.norm()), d / float(w.grad.norm())
    rs.close()


@pytest.mark.gpu
def test_training_repeats_bit_for_bit():
    import torch
    from flash5_b200.riemann import ExactRiemann
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    X = torch.randn(12345, 8, generator=g, device="cuda")
    T = torch.randn(12345, generator=g, device="cuda")
    out = []
    for _ in range(2):
        rs = ExactRiemann(device=0)
        loss = rs.train(X, T, 12345, epochs=2, batch=1000)
        out.append((rs.weights(), loss))
        rs.close()
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
