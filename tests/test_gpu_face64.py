"""The FP64 face work with branch-free divisions and square roots, and its way
back to the plain form where an operand leaves their range: fluxes of a block
whose cells span ordinary, slow (the divisor 1 - v^2 c^2 rounds to a
significand of all ones), zero and extreme values equal the CPU oracle's bit
for bit, for PLM and PPM, staged and not."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage", [0, 1])
@pytest.mark.parametrize("limiter", ["mc", "ppm"])
def test_fluxes_equal_the_oracle(limiter, stage):
    from bhgpu import fixed as fx
    from bhgpu.fixed import FxGrid, FxParams
    from oracle import fixed as ofx
    p = FxParams(precision="fp64", limiter=limiter)
    # 8^3 cells of 1/8 from -1/2: the disc inside the ring singularity among the face centres
    blocks = FxGrid.uniform(-4.0, 4.0, 64, 64, p) if stage else FxGrid.uniform(-0.5, 0.5, 8, 8, p)
    g = blocks
    h = ofx.FxHost(g.blocks_np, g.nbr_np, ofx.params(p))
    rng = np.random.default_rng(5)
    N = g.ncell
    W = np.zeros((8, N))
    W[0] = 10 ** rng.uniform(-12, 2, N)
    W[1] = W[0] * 10 ** rng.uniform(-6, 2, N)
    W[2:5] = rng.normal(size=(3, N)) * 10 ** rng.uniform(-12, 1, N)
    W[5:8] = rng.normal(size=(3, N)) * 10 ** rng.uniform(-12, 1, N)
    kind = rng.integers(0, 12, N)
    W[2:5, kind == 0] = 0.0
    W[5:8, kind == 1] = 0.0
    W[2:5, kind == 2] = 1e-8 * rng.normal(size=(3, int((kind == 2).sum())))
    W[:2, kind == 3] *= 1e-150                      # below the range
    W[2:5, kind == 4] = 1e7 * rng.normal(size=(3, int((kind == 4).sum())))   # beyond it
    Bf = rng.normal(size=(3, N)) * 10 ** rng.uniform(-12, 0, N)
    g.W.copy_(torch.as_tensor(W))
    g.Bf.copy_(torch.as_tensor(Bf))
    h.W[:], h.Bf[:] = W, Bf
    before = fx.tune_get("fp64", "stage")
    fx.tune_set("fp64", "stage", stage)
    try:
        g.fluxes(0)
    finally:
        fx.tune_set("fp64", "stage", before)
    h.fluxes(0)
    F, Fh = g.F.cpu().numpy(), np.array(h.F).reshape(g.F.shape)
    assert np.array_equal(F, Fh, equal_nan=True)
