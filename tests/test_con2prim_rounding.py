"""The faithful con2prim's shortcuts -- the residual's sign without its value,
the bracket's growth and the Newton cycle without their evaluations, the
divisions without a branch -- give the bits of the plain loops.

On the CPU the host build of the kernels' con2prim is compared with the C
restatement of the reference's (oracle), whose loops have none of them, over
the stress batch's ranges and over states without physics in them: random
magnitudes and signs, zeros, NaN and infinities, tau far below zero (the
bracket runs away to overflow) and near-static gas (cells that cannot reach
the tolerance).  On the GPU a batch is compared with the same cells in
batches of other sizes (the lanes of a warp then take other cells up), and
with the oracle where its metric is exact (flat space)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from bhgrid import configs


def states(kind, n, seed):
    rng = np.random.default_rng(seed)
    r, th = rng.uniform(1.5, 50.0, n), np.arccos(rng.uniform(-1, 1, n))
    if kind == "wild":
        U = 10 ** rng.uniform(-12, 12, (8, n)) * rng.choice([-1.0, 1.0], (8, n))
        U[0] = np.where(rng.random(n) < 0.9, np.abs(U[0]), U[0])
        for v in (0.0, np.nan, np.inf):
            m = rng.random((8, n)) < 0.005
            U[m] = v
    elif kind == "negative tau":
        U = rng.normal(size=(8, n))
        U[0] = 10 ** rng.uniform(-6, 4, n)
        U[4] = -10 ** rng.uniform(-2, 6, n)
    elif kind == "static":
        U = 1e-9 * rng.normal(size=(8, n))
        U[0] = 10 ** rng.uniform(-3, 6, n)
        U[4] = U[0] * 10 ** rng.uniform(-3, 2, n)
    else:
        W, r, th = configs.con2prim_batch(n, seed=seed)
        U = oracle.Oracle(1.0, 0.9375, 0.0, 4.0 / 3.0).ptoc(W, r, th)[0]
    return np.ascontiguousarray(U), r, th



def eq(a, b):
    return np.array_equal(a, b, equal_nan=True)


KINDS = ("stress", "wild", "negative tau", "static")


@pytest.mark.parametrize("M,a", [(0.0, 0.0), (1.0, 0.9375)])
@pytest.mark.parametrize("kind", KINDS)
def test_host_build_equals_the_plain_loops(kind, M, a):
    from hostcheck import HostKernels
    n = 20000
    U, r, th = states(kind, n, 7)
    orc = oracle.Oracle(M, a, 0.0, 4.0 / 3.0)
    hk = HostKernels(M, a, 0.0, 4.0 / 3.0, 1)
    W, Wd = np.zeros((8, n)), np.zeros((5, n))
    st, it, pa = (np.zeros(n, np.int32) for _ in range(3))
    d = lambda x: C.c_void_p(x.ctypes.data)  # noqa: E731
    hk.call("hc_ctop", d(U), d(r), d(th), C.c_int64(n), d(W), d(Wd), d(st), d(it), d(pa))
    Wc, Wdc, stc, itc, pac = orc.ctop(U, r, th)
    assert np.array_equal(st, stc) and np.array_equal(it, itc) and np.array_equal(pa, pac)
    ok = st == 1
    assert eq(W[:, ok], Wc[:, ok]) and eq(Wd[:, ok], Wdc[:, ok])
    if kind == "stress" and M:
        assert (it == 500).any() and (pa == 3).any()   # the cases the shortcuts are for


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 4 * 148 * 128 + 1])
def test_batches_of_any_size_give_the_same_bits(n):
    import torch
    import bhgpu
    U, r, th = (torch.as_tensor(x, device="cuda") for x in states("stress", n, 3))
    cn = bhgpu.Conserved(bhgpu.Metric(1.0, 0.9375), bhgpu.State(4.0 / 3.0))
    whole = cn.ctop(U, r, th, check_domain=False)
    for lo in list(range(0, n, max(1, n // 3)))[:4]:
        hi = min(n, lo + 97)
        part = cn.ctop(U[:, lo:hi].contiguous(), r[lo:hi].contiguous(), th[lo:hi].contiguous(), check_domain=False)
        for x, y in zip(whole[2:], part[2:]):
            assert torch.equal(x[lo:hi], y)
        ok = part[2] == 1
        for x, y in zip(whole[:2], part[:2]):
            assert eq(x[:, lo:hi][:, ok].cpu().numpy(), y[:, ok].cpu().numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_device_equals_the_plain_loops_in_flat_space(kind):
    """In flat space at the same (r, theta) the device and the host differ by
    sin/cos of theta alone: theta = pi/2 exactly on both sides."""
    import torch
    import bhgpu
    n = 20000
    U, r, _ = states(kind, n, 11)
    th = np.full(n, np.pi / 2)
    r = np.ones(n)
    orc = oracle.Oracle(0.0, 0.0, 0.0, 4.0 / 3.0)
    cn = bhgpu.Conserved(bhgpu.Metric(0.0, 0.0), bhgpu.State(4.0 / 3.0))
    W, Wd, st, it, pa = (x.cpu().numpy() for x in cn.ctop(U, r, th, check_domain=False))
    Wc, Wdc, stc, itc, pac = orc.ctop(U, r, th)
    assert np.array_equal(st, stc) and np.array_equal(it, itc) and np.array_equal(pa, pac)
    ok = st == 1
    assert eq(W[:, ok], Wc[:, ok]) and eq(Wd[:, ok], Wdc[:, ok])
