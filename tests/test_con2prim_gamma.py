"""The faithful con2prim's sign shortcuts rest on Gamma > 1 (the pressure's
factor (Gamma - 1) / Gamma is then positive).  bh_ctop takes any Gamma: at and
below 1 it gives the plain loops' bits too -- the host build of the kernels
against the C restatement, and the device in flat space."""
import ctypes as C

import numpy as np
import pytest

import oracle
from test_con2prim_rounding import KINDS, eq, states

GAMMAS = (0.05, 0.3, 0.6, 0.9, 1.0, 1.05, 50.0)


@pytest.mark.parametrize("gamma", GAMMAS)
@pytest.mark.parametrize("kind", KINDS)
def test_host_build_equals_the_plain_loops(kind, gamma):
    from hostcheck import HostKernels
    n = 20000
    U, r, th = states(kind, n, 7)
    orc = oracle.Oracle(1.0, 0.9375, 0.0, gamma)
    hk = HostKernels(1.0, 0.9375, 0.0, gamma, 1)
    W, Wd = np.zeros((8, n)), np.zeros((5, n))
    st, it, pa = (np.zeros(n, np.int32) for _ in range(3))
    d = lambda x: C.c_void_p(x.ctypes.data)  # noqa: E731
    hk.call("hc_ctop", d(U), d(r), d(th), C.c_int64(n), d(W), d(Wd), d(st), d(it), d(pa))
    Wc, Wdc, stc, itc, pac = orc.ctop(U, r, th)
    assert np.array_equal(st, stc) and np.array_equal(it, itc) and np.array_equal(pa, pac)
    ok = st == 1
    assert eq(W[:, ok], Wc[:, ok]) and eq(Wd[:, ok], Wdc[:, ok])


@pytest.mark.gpu
@pytest.mark.parametrize("gamma", GAMMAS)
@pytest.mark.parametrize("kind", KINDS)
def test_device_equals_the_plain_loops_in_flat_space(kind, gamma):
    import bhgpu
    n = 20000
    U, _, _ = states(kind, n, 11)
    r, th = np.ones(n), np.full(n, np.pi / 2)
    orc = oracle.Oracle(0.0, 0.0, 0.0, gamma)
    cn = bhgpu.Conserved(bhgpu.Metric(0.0, 0.0), bhgpu.State(gamma))
    W, Wd, st, it, pa = (x.cpu().numpy() for x in cn.ctop(U, r, th, check_domain=False))
    Wc, Wdc, stc, itc, pac = orc.ctop(U, r, th)
    assert np.array_equal(st, stc) and np.array_equal(it, itc) and np.array_equal(pa, pac)
    ok = st == 1
    assert eq(W[:, ok], Wc[:, ok]) and eq(Wd[:, ok], Wdc[:, ok])
