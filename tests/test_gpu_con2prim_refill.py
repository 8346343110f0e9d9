"""con2prim batches whose warps take cells up again and again (more cells than
the resident lanes), with an odd remainder: every cell equals the same cell in
chunks in which each lane has one cell, with and without a given start, and
the C restatement in flat space."""
import numpy as np
import pytest

import oracle
from test_con2prim_rounding import eq, states

pytestmark = pytest.mark.gpu


def one_wave():
    """cells that a launch spreads as one per lane: 4 CTAs of 128 per SM"""
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 4 * 128


def mixed_states(n, seed):
    """stress cells with cells without physics in them strewn in, so that
    neighbours end after very different counts"""
    parts = [states(k, m, seed) for k, m in (("stress", n - n // 5), ("wild", n // 10),
                                             ("negative tau", n // 5 - n // 10))]
    order = np.random.default_rng(seed).permutation(n)
    return [np.ascontiguousarray(np.concatenate([p[i] for p in parts], axis=-1)[..., order]) for i in range(3)]


def same(whole, part, lo, hi):
    import torch
    for x, y in zip(whole[2:], part[2:]):
        assert torch.equal(x[lo:hi], y)
    ok = part[2] == 1
    for x, y in zip(whole[:2], part[:2]):
        assert eq(x[:, lo:hi][:, ok].cpu().numpy(), y[:, ok].cpu().numpy())


@pytest.mark.parametrize("start", [False, True])
@pytest.mark.parametrize("waves,rest", [(1, 1), (2, 17), (6, 33), (25, 101)])
def test_refilled_lanes_give_each_cells_bits(waves, rest, start):
    import torch
    import bhgpu
    from bhgpu.c2p_guess import C2PGuess
    wave = one_wave()
    n = waves * wave + rest
    U, r, th = (torch.as_tensor(x, device="cuda") for x in mixed_states(n, 5))
    cn = bhgpu.Conserved(bhgpu.Metric(1.0, 0.9375), bhgpu.State(4.0 / 3.0))
    if start:
        g = C2PGuess(cn)
        xi0 = torch.as_tensor(10 ** np.random.default_rng(8).uniform(-6, 6, n), device="cuda")
        xi0[::7] = float("nan")
        run = lambda lo, hi: g.ctop_from(U[:, lo:hi].contiguous(), r[lo:hi].contiguous(),  # noqa: E731
                                         th[lo:hi].contiguous(), xi0[lo:hi].contiguous())
    else:
        run = lambda lo, hi: cn.ctop(U[:, lo:hi].contiguous(), r[lo:hi].contiguous(),  # noqa: E731
                                     th[lo:hi].contiguous(), check_domain=False)
    whole = run(0, n)
    for lo in range(0, n, wave):
        same(whole, run(lo, min(n, lo + wave)), lo, min(n, lo + wave))


def test_refilled_lanes_equal_the_plain_loops_in_flat_space():
    import bhgpu
    n = 3 * one_wave() + 77
    U, _, _ = mixed_states(n, 13)
    r, th = np.ones(n), np.full(n, np.pi / 2)
    cn = bhgpu.Conserved(bhgpu.Metric(0.0, 0.0), bhgpu.State(4.0 / 3.0))
    W, Wd, st, it, pa = (x.cpu().numpy() for x in cn.ctop(U, r, th, check_domain=False))
    Wc, Wdc, stc, itc, pac = oracle.Oracle(0.0, 0.0, 0.0, 4.0 / 3.0).ctop(U, r, th)
    assert np.array_equal(st, stc) and np.array_equal(it, itc) and np.array_equal(pa, pac)
    ok = st == 1
    assert eq(W[:, ok], Wc[:, ok]) and eq(Wd[:, ok], Wdc[:, ok])
