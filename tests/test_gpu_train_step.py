"""The training step's kernels (k_train, k_train_reduce) at the edges of their
tiles: batches of one cell, around one tile of 64 cells (a single partial
gradient, written in place, against several) and of more tiles than CTAs,
against the CPU restatement (oracle/mlp.py, FP64)."""
import numpy as np
import pytest
import torch

from oracle import mlp

pytestmark = pytest.mark.gpu

# A gradient component is a sum over the cells of delta x activation; a
# delta's rounding is at most that of the sums it comes through -- 6 + 64 +
# 64 forward terms, 2 + 64 backward, and as many roundings again in the
# sums over cells, tanh included: under 340 roundings of 2^-24 = 2e-5 of the
# sum of the terms' magnitudes (|delta| from the magnitudes of its own terms).
TOL = 2e-5


@pytest.mark.parametrize("n", [1, 17, 63, 64, 65, 1000, 64 * 300 + 5])
def test_gradient_at_tile_edges(n):
    import bhgpu
    rng = np.random.default_rng(n)
    cn = bhgpu.Conserved(bhgpu.Metric(1.0, 0.9375, 0.0), bhgpu.State(4.0 / 3.0))
    g = bhgpu.C2PGuess(cn, seed=3)
    pre = np.stack([10 ** rng.uniform(-6, 2, n), 10 ** rng.uniform(-6, 2, n), 10 ** rng.uniform(-6, 2, n),
                    10 ** rng.uniform(-6, 2, n), rng.normal(size=n)])
    r = rng.uniform(1.5, 50.0, n)
    x = mlp.features(pre, r)
    w = g.w.cpu().numpy()
    w[mlp.NPARAM:mlp.NPARAM + 6] = [0.0, 1.0, 2.0, 1.0, 0.0, 3.0]
    w[mlp.NPARAM + 6:] = [0.2, 0.3, 0.1, 0.3, 0.5, 1.0]
    g.w.copy_(torch.as_tensor(w))
    tgt = rng.normal(size=(2, n)).astype(np.float32)
    dev = [torch.as_tensor(a, device="cuda") for a in (pre, r, tgt)]
    before = g.w.clone()
    L, grad = g.gradient(*dev)
    assert torch.equal(g.w, before)                 # lr = 0 only computes
    wf = g.w.double().cpu().numpy()
    Lc, gc = mlp.loss_and_grad(wf, x, tgt.T.astype(np.float64))
    # the sums of magnitudes: every weight, activation and error by its size
    p = mlp.unpack(wf)
    xn, h1, h2, y = (np.abs(a) for a in mlp.forward(wf, x))
    W2, W3 = np.abs(mlp.bf16(p["W2"])), np.abs(mlp.bf16(p["W3"]))
    mag = h2 @ W3.T + np.abs(mlp.bf16(p["b3"])) + np.abs(tgt.T)
    dy = 2.0 * mag / n
    d2 = dy @ W3
    d1 = d2 @ W2
    a = {"W1": d1.T @ xn, "b1": d1.sum(0), "W2": d2.T @ h1, "b2": d2.sum(0), "W3": dy.T @ h2, "b3": dy.sum(0)}
    bound = TOL * np.concatenate([a[k].reshape(-1) for k, _ in mlp.SIZES])
    assert (np.abs(grad - gc) <= bound).all()
    assert abs(L - Lc) <= TOL * float((2.0 * mag * mag).sum())
