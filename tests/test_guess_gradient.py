"""The network's parameter gradient at the row counts and feature counts where its split over warps and
blocks changes (a partial warp, a partial block, one block, several rounds of all blocks), against the
FP64 oracle. Every sum is of FP32 products in chains of at most a few hundred terms: the error bound is
1e-4 of the largest entry, that of the existing comparison at 3,000 rows and 4 features."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize('F', [1, 3, 4, 5, 8])
@pytest.mark.parametrize('rows', [1, 31, 33, 256, 257, 77824, 100003])
def test_gradient_over_rows_and_features(gpu_lib, F, rows):
    import torch
    from opencmp_gb300.guess import GuessNet
    from oracle import mlp
    rng = np.random.default_rng(100 * F + rows)
    net = GuessNet(F, seed=1)
    P = (rng.standard_normal(net.nparams) * 0.3).astype(np.float32)
    net.set_params(P)
    X = rng.standard_normal((rows, F)).astype(np.float32)
    T = rng.standard_normal(rows).astype(np.float32)
    Xd = torch.as_tensor(X, device='cuda')
    loss, g = net.loss_grad(Xd, torch.as_tensor(T, device='cuda'), want_grad=True)
    lo, go = mlp.loss_grad(P.astype(np.float64), X.astype(np.float64), T.astype(np.float64))
    assert abs(loss - lo) <= 1e-5 * lo
    assert np.abs(g - go).max() <= 1e-4 * np.abs(go).max()
    dY = (rng.standard_normal(rows) * 1e-2).astype(np.float32)
    gb = net.backward(Xd, torch.as_tensor(dY, device='cuda'), want_grad=True)
    gbo = mlp.backward(P.astype(np.float64), X.astype(np.float64), dY.astype(np.float64))
    assert np.abs(gb - gbo).max() <= 1e-4 * np.abs(gbo).max()
    _, g2 = net.loss_grad(Xd, torch.as_tensor(T, device='cuda'), want_grad=True)
    assert g.tobytes() == g2.tobytes()
