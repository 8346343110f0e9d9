"""The library's own choice of launch bounds, staging and update form
(bh_fx_tune_set's initial values) on both sides of each of its rules: few
items and many, tiles that pad by more and by less than a tenth, one level
and several, PLM and PPM.  FP64 without contraction gives the same bits
whatever is chosen, so a step equals one with the plain kernels (no register
cap, unstaged, one update kernel)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def grid(case, limiter):
    from bhgpu.fixed import FxGrid, FxParams
    from bhgrid.blocks import torus_levels
    p = FxParams(precision="fp64", limiter=limiter)
    if case == "levels":
        return FxGrid.leveled(-40.0, 40.0, torus_levels(nb=8, r_fine=(14.0, 26.0), seed=3), 4, p, persistent=True)
    return FxGrid.uniform(-40.0, 40.0, case[0], case[1], p)


@pytest.mark.parametrize("limiter", ["mc", "ppm"])
@pytest.mark.parametrize("case", [(16, 8), (32, 32), (64, 64), (96, 24), (104, 104), "levels"])
def test_step_does_not_depend_on_the_choice(case, limiter):
    from bhgpu import fixed as fx
    a, b = grid(case, limiter), grid(case, limiter)
    before = {k: fx.tune_get("fp64", k) for k in fx.TUNE_KNOBS}
    try:
        for k in fx.TUNE_KNOBS:
            fx.tune_set("fp64", k, 2 if k in ("stage", "split") else 0)
        a.torus_init(seed=2)
        for _ in range(2):
            a.step()
        for k in fx.TUNE_KNOBS:
            fx.tune_set("fp64", k, 0 if k in ("stage", "split") else 1)
        b.torus_init(seed=2)
        for _ in range(2):
            b.step()
    finally:
        for k, v in before.items():
            fx.tune_set("fp64", k, v)
    for name in ("U", "W", "Bf", "dt"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
