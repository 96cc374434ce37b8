"""Sweep calls that follow one another on one grid: what a call keeps for the
next (plan, item list, captured launches) has to fit the next call's own sweep
count, active set and levels.  Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_grid import random_sparse
from test_gpu_sweep import assert_same_blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsx", [8, 16])
@pytest.mark.parametrize("stencil", [0, 1])
def test_sweep_counts_in_turn(msbg, ctx, oracle, bsx, stencil):
    """More sweeps than before and fewer again: the second call of a count
    runs what the buffers of that moment hold."""
    host = random_sparse(msbg, 4 * bsx, 4 * bsx, 4 * bsx, bsx, 0.7, 19 + stencil, empty=0.1, full=0.9)
    active = sorted(host.blocks)
    dev = msbg.SparseGrid.from_host(ctx, host)
    sw = msbg.Sweeper(dev)
    for iterations in (2, 40, 2, 1, 150, 40, 2, 1):
        sw.sweep(active, stencil, msbg.PdeParams(0.02, iterations, False))
        oracle.sweep(host, active, stencil, 0.02, iterations, False)
        assert_same_blocks(dev, host, np.arange(host.n_blocks))


def test_coarse_level_made_anew(msbg, ctx, oracle):
    """A coarse level that is destroyed and made again, with its blocks in
    another order or with other blocks: often the same address, as many calls
    on it and as many slots, but not the slots an earlier plan names."""
    sx, sy, sz = 64, 48, 80
    r = np.random.default_rng(4)
    fine = msbg.HostGrid("fine", sx, sy, sz, 0.0, 0.0, 16)
    levels = (r.random(fine.n_blocks) < 0.5).astype(np.uint8)
    active = [b for b in range(fine.n_blocks) if levels[b] == 0]
    for b in active:
        fine.ensure_block(b)
        fine.blocks[b][:] = r.uniform(0, 1, 4096)
    dfine = msbg.SparseGrid.from_host(ctx, fine)
    sw = msbg.Sweeper(dfine)
    of_level = [b for b in range(fine.n_blocks) if levels[b] == 1]
    for turn in range(8):
        ids = np.sort(r.permutation(of_level)[:-3]) if turn % 2 else np.array(of_level[:-3])
        ids = r.permutation(ids).astype(np.uint64)
        coarse = msbg.HostGrid("coarse", sx // 2, sy // 2, sz // 2, 0.0, 0.0, 8)
        for b in ids:
            coarse.ensure_block(int(b))
            coarse.blocks[int(b)][:] = r.uniform(0, 1, 512)
        dcoarse = msbg.SparseGrid(ctx, sx // 2, sy // 2, sz // 2, 0.0, 0.0, 8)
        dcoarse.write_blocks(ids, np.stack([coarse.blocks[int(b)] for b in ids]))
        sw.sweep_multires(dcoarse, levels, active, 1, msbg.PdeParams(0.05, 1, False))
        ctx.synchronize()
        oracle.sweep_multires(fine, coarse, levels, active, 1, 0.05, 1, False)
        assert_same_blocks(dfine, fine, active)
        dcoarse.close()
