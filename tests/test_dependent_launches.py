"""The corrected scheme's step kernels run as programmatic dependents: a
kernel is resident while the one before it still writes.  On the CPU the
source is held to what that asks for (every kernel so launched waits before
anything else, and none reads through the non-coherent path); on the GPU the
steps in a stream, which are launched so, equal a graph's replays, which are
not."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "black-hole-simulator_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def launched():
    """names of the kernels launched by fx_launch"""
    return sorted(set(re.findall(r"fx_launch\(fx::(k_\w+)", source("bh_fixed.cuh"))))


def test_every_dependent_kernel_waits_first():
    text = source("bh_fixed.cuh")
    names = launched()
    assert len(names) >= 8
    for k in names:
        body = re.search(r"\b" + k + r"\([^{;]*\)\s*\{\s*([^;]*;)", text)
        assert body and body.group(1) == "after_previous();", k


@pytest.mark.parametrize("name", ["bh_fixed.cuh", "bh_fixed_phys.cuh", "bh_div.cuh"])
def test_no_load_through_the_non_coherent_path(name):
    assert not re.findall(r"__ldg|ld\.global\.nc|__restrict__|__ldlu|tex1Dfetch", source(name))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp64-fma", "mixed"])
@pytest.mark.parametrize("case", [(16, 16, False), (64, 64, False), (72, 24, True), "levels"])
def test_stream_equals_graph(case, precision):
    import torch
    from bhgpu.fixed import FxGrid, FxParams
    from bhgrid.blocks import torus_levels

    def grid():
        p = FxParams(precision=precision)
        if case == "levels":
            return FxGrid.leveled(-40.0, 40.0, torus_levels(nb=6, r_fine=(14.0, 26.0), seed=3), 4, p, persistent=True)
        return FxGrid.uniform(-40.0, 40.0, case[0], case[1], p, persistent=case[2])
    a, b = grid(), grid()
    a.torus_init(seed=4)
    b.torus_init(seed=4)
    for _ in range(6):
        a.step()
    b.capture()
    for _ in range(6):
        b.replay()
    torch.cuda.synchronize()
    for name in ("U", "W", "Bf", "dt"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
    b.release_graph()
