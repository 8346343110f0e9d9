"""The mixed variant by the library's launch rules against the plain kernels
(no register cap, unstaged, one update kernel), on both sides of the rules'
lines.  The variant contracts multiply-adds, so kernels may round differently;
a step's state agrees to FP32 rounding of the fluxes (relative to each array's
largest value 2^-22 per step)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limiter", ["mc", "ppm"])
@pytest.mark.parametrize("case", [(16, 8), (40, 40), (48, 48), (96, 24), (128, 128), "levels"])
def test_rules_against_plain_kernels(case, limiter):
    from bhgpu import fixed as fx
    from bhgrid.blocks import torus_levels
    p = fx.FxParams(precision="mixed", limiter=limiter)
    out = []
    for rules in (True, False):
        for k in fx.TUNE_KNOBS:
            form = k in ("stage", "split")
            fx.tune_set("mixed", k, (2 if form else 0) if rules else (0 if form else 1))
        g = (fx.FxGrid.leveled(-40.0, 40.0, torus_levels(nb=8, r_fine=(14.0, 26.0), seed=3), 4, p, persistent=True)
             if case == "levels" else fx.FxGrid.uniform(-40.0, 40.0, case[0], case[1], p))
        g.torus_init(seed=2)
        for _ in range(2):
            g.step()
        out.append(g)
    for name in ("U", "W", "Bf"):
        a, b = (getattr(g, name).double() for g in out)
        scale = a.abs().amax(1, keepdim=True)
        assert ((a - b).abs() <= 2 * 2.0 ** -22 * scale).all(), name
