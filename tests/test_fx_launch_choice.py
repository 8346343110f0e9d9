"""What the corrected scheme's launch rules take, on both sides of each line
(bh_fx_tune_choice: host code, no launch), and on the GPU that a grid whose
tiles fit exactly runs the staged fluxes with the same bits."""
import ctypes as C

import numpy as np
import pytest

KNOBS = ("c2p", "flux", "update", "stage", "split")


def choice(knob, precision, counts, limiter="mc"):
    from bhgpu.fixed import BhFxGrid, FxParams, lib
    g = BhFxGrid()
    g.nitem_cell, g.nitem_pos, g.nitem_flux, g.rule_tile = (counts[k] for k in ("cell", "pos", "flux", "tile"))
    p, v = FxParams(precision=precision, limiter=limiter).cstruct(), C.c_int32(-1)
    assert lib.bh_fx_tune_choice(C.byref(p), C.byref(g), KNOBS.index(knob), C.byref(v)) == 0
    return v.value


def counts(n, nb=1, **kw):
    from bhgrid.blocks import item_counts
    blocks = np.zeros(nb ** 3, [("n", "<i4")])
    blocks["n"] = n
    return item_counts(blocks, **kw)


@pytest.fixture(autouse=True)
def by_rule():
    from bhgpu import fixed as fx
    before = {(p, k): fx.tune_get(p, k) for p in fx.PRECISIONS for k in fx.TUNE_KNOBS}
    for p, k in before:
        fx.tune_set(p, k, 2 if k in ("stage", "split") else 0)
    yield
    for (p, k), v in before.items():
        fx.tune_set(p, k, v)


@pytest.mark.parametrize("n,nb,mixed,fp64,fma", [
    (48, 2, 0, 0, 0),      # below TILE_MIN: no tiles, the lists equally long
    (126, 1, 1, 1, 1),     # exact fits: the lists equally long, all tiles
    (110, 1, 1, 1, 0), (102, 1, 1, 1, 0), (94, 1, 0, 0, 0), (70, 1, 0, 0, 0), (70, 2, 1, 1, 1),
    (64, 2, 0, 0, 0),      # padded by 16 %
    (104, 1, 0, 0, 0), (124, 1, 1, 1, 0), (128, 1, 1, 1, 0), (92, 2, 1, 1, 0)])
def test_staging(n, nb, mixed, fp64, fma):
    c = counts(n, nb)
    assert [choice("stage", p, c) for p in ("mixed", "fp64", "fp64-fma")] == [mixed, fp64, fma]
    assert all(choice("stage", p, c, "ppm") == 0 for p in ("mixed", "fp64", "fp64-fma"))


def test_a_list_without_tiles_is_not_staged():
    for n in (64, 126):
        c = counts(n, tile_min=1000)
        assert c["flux"] == c["pos"] and c["tile"] == 0
        assert all(choice("stage", p, c) == 0 for p in ("mixed", "fp64", "fp64-fma"))


def test_grids_bring_their_tiles():
    from bhgpu.fixed import FxGrid, FxParams
    g = FxGrid.leveled(-1.0, 1.0, np.zeros((1, 1, 1), np.int32), 70, FxParams(), device="cpu")
    assert g._g.nitem_flux == g._g.nitem_pos == g._g.rule_tile == 2916


def test_caps_where_the_uncapped_kernels_would_queue():
    """no cap up to the CTAs the uncapped kernels keep resident: 2 per SM in
    FP64, 4 in FP32 (a host without a GPU counts as one SM)"""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 1
    for prec, per_sm, caps in (("mixed", 4, (7, 8, 8)), ("fp64", 2, (6, 5, 4)), ("fp64-fma", 2, (6, 5, 4))):
        for items, want in ((per_sm * sms, (1, 1, 1)), (per_sm * sms + 1, caps)):
            c = dict(cell=items, pos=items, flux=items, tile=0)
            assert tuple(choice(k, prec, c) for k in ("c2p", "flux", "update")) == want
            c["cell"] = 1     # (each kernel by its own list)
            assert (choice("c2p", prec, c), choice("flux", prec, c)) == (1, want[1])


def test_two_update_kernels_where_one_takes_more_waves():
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 1
    for prec, per_sm in (("mixed", 16), ("fp64", 4), ("fp64-fma", 4)):
        for items, want in ((per_sm * sms, 0), (per_sm * sms + 1, 1)):
            assert choice("split", prec, dict(cell=items, pos=items, flux=items, tile=0)) == want


@pytest.mark.gpu
def test_exact_tiles_take_the_staged_fluxes_with_the_same_bits():
    import torch
    from bhgpu import fixed as fx
    out = []
    for stage in (2, 0):
        fx.tune_set("fp64", "stage", stage)
        g = fx.FxGrid.leveled(-40.0, 40.0, np.zeros((1, 1, 1), np.int32), 102, fx.FxParams(precision="fp64"))
        assert g.launch_choice("stage") == (1 if stage == 2 else 0)
        g.torus_init(seed=2)
        for _ in range(2):
            g.step()
        out.append(g)
    for name in ("U", "W", "Bf", "dt"):
        assert torch.equal(getattr(out[0], name), getattr(out[1], name)), name
