"""The launch rules on a sharded domain: every rank takes the same kernels,
however its work lists differ in length (the contracted variants' kernels
round differently, and a face shared by two ranks is computed by both)."""
import os
import socket
import tempfile
from datetime import timedelta

import numpy as np
import pytest
import torch
import torch.multiprocessing as mp

KNOBS = ("c2p", "flux", "update", "stage", "split")


def test_item_counts_are_the_lists_lengths():
    from bhgrid.blocks import flux_items, item_counts, leveled_blocks, torus_levels, uniform_blocks, work_items
    cases = [uniform_blocks(-1.0, 1.0, 64, 64)[0], uniform_blocks(-1.0, 1.0, 24, 8)[0],
             leveled_blocks(-40.0, 40.0, torus_levels(nb=6, r_fine=(14.0, 26.0), seed=3), 10)[0]]
    for blocks in cases:
        for tile_min in (16, 64):
            c = item_counts(blocks, tile_min)
            assert c["cell"] == len(work_items(blocks, "cell")) and c["pos"] == len(work_items(blocks, "pos"))
            flux = flux_items(blocks, tile_min)
            assert c["flux"] == len(flux) and c["tile"] == (flux[:, 1] >= 0).sum()


def _worker(rank, world, port, out_dir):
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    sys.path.insert(0, os.path.join(os.path.dirname(here), "black-hole-simulator_b200"))
    import torch.distributed as dist
    from bhgpu.fixed import FxGrid, FxParams
    from bhgpu.fxshard import ShardedFxGrid
    from bhgrid.blocks import uniform_blocks
    os.environ["MASTER_ADDR"], os.environ["MASTER_PORT"] = "127.0.0.1", str(port)
    dist.init_process_group("gloo", rank=rank, world_size=world, timeout=timedelta(seconds=120))
    try:
        blocks, nbr = uniform_blocks(-40.0, 40.0, 32, 8)
        owner = np.ones(len(blocks), np.int32)
        owner[:1] = 0                                    # 4 work items of cells against 252
        got = []
        for prec in ("fp64", "fp64-fma", "mixed"):
            prm = FxParams(precision=prec)
            sh = ShardedFxGrid(blocks, nbr, lambda lb, ln, na, ml: FxGrid(lb, ln, prm, device="cpu", nactive=na,
                                                                          maxlevel=ml), owner=owner)
            alone = FxGrid(sh.local.blocks, sh.local.nbr, prm, device="cpu", nactive=sh.local.nown)
            got.append([[g.launch_choice(k) for k in KNOBS] for g in (sh.grid, alone)])
        np.save(os.path.join(out_dir, f"r{rank}.npy"), np.array(got))
    finally:
        dist.destroy_process_group()


def test_ranks_of_unequal_shares_choose_the_same_kernels():
    s = socket.socket()
    s.bind(("127.0.0.1", 0))
    port = s.getsockname()[1]
    s.close()
    with tempfile.TemporaryDirectory() as d:
        mp.start_processes(_worker, args=(2, port, d), nprocs=2, join=True, start_method="spawn")
        a, b = (np.load(os.path.join(d, f"r{r}.npy")) for r in range(2))
    assert np.array_equal(a[:, 0], b[:, 0])
    # the case is one where each rank's own lists would choose otherwise (on a
    # host without a GPU the rules count on one SM)
    if not torch.cuda.is_available():
        assert not np.array_equal(a[:, 1], b[:, 1])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp64-fma", "mixed"])
def test_unequal_shares_step_as_the_whole_grid(precision):
    """Two local grids (one block of 32^3, and the 26 others) stepped piece by
    piece in one process, the copies' boxes moved between the pieces as
    ShardedFxGrid does, equal the whole grid bit for bit."""
    from bhgpu.fixed import FxGrid, FxParams
    from bhgrid.blocks import box_size, uniform_blocks
    from bhgrid.shard import local_grid
    prm = FxParams(precision=precision)
    blocks, nbr = uniform_blocks(-40.0, 40.0, 96, 32)
    whole = FxGrid(blocks, nbr, prm)
    whole.torus_init(seed=6)
    owner = np.ones(len(blocks), np.int32)
    owner[13] = 0                                        # the block around the hole
    loc = [local_grid(blocks, nbr, owner, r) for r in range(2)]
    grids = [FxGrid(lg.blocks, lg.nbr, prm, nactive=lg.nown) for lg in loc]
    for g in grids:
        g.launch_as_share_of(blocks, 2)
    assert [grids[0].launch_choice(k) for k in KNOBS] == [grids[1].launch_choice(k) for k in KNOBS]
    box = box_size(32)
    where = [{int(g): i for i, g in enumerate(lg.glob)} for lg in loc]

    def put(name, dst, d, src, s):
        getattr(dst, name)[:, d:d + box].copy_(getattr(src, name)[:, s:s + box])

    for r, lg in enumerate(loc):
        for i, g in enumerate(lg.glob):
            for name in ("U", "W", "Bf"):
                put(name, grids[r], int(lg.blocks["off"][i]), whole, int(blocks["off"][g]))

    def exchange(names):
        for r, lg in enumerate(loc):
            for i in range(lg.nown, len(lg.glob)):
                j = where[1 - r][int(lg.glob[i])]
                for name in names:
                    put(name, grids[r], int(lg.blocks["off"][i]), grids[1 - r], int(loc[1 - r].blocks["off"][j]))

    for _ in range(3):
        whole.step()
        for stage in (0, 1):
            for g in grids:
                g.prims(stage, with_dt=stage == 0)
            if stage == 0:
                dt = torch.minimum(grids[0].dt[:1], grids[1].dt[:1]).clone()
                for g in grids:
                    g.dt[:1].copy_(dt)
            exchange(("W", "Bf1" if stage else "Bf"))
            for g in grids:
                g.ghost_pass(stage, 0)
            for g in grids:
                g.fluxes(stage)
            for g in grids:
                g.update(stage)
    for r, lg in enumerate(loc):
        for i in range(lg.nown):
            lo, go = int(lg.blocks["off"][i]), int(blocks["off"][lg.glob[i]])
            for name in ("U", "Bf"):
                a = getattr(grids[r], name)[:, lo:lo + box].view(-1, 39, 39, 39)[:, 3:35, 3:35, 3:35]
                b = getattr(whole, name)[:, go:go + box].view(-1, 39, 39, 39)[:, 3:35, 3:35, 3:35]
                assert torch.equal(a, b), (name, int(lg.glob[i]))
