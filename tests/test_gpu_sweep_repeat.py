"""Sweep calls that follow one another on one grid: what a call keeps for the
next (plan, item list, captured launches) has to fit the next call's own sweep
count, active set and levels.  Bit for bit against the oracle."""
import time

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


def test_few_blocks_of_a_tall_domain(msbg, ctx):
    """Blocks near the top of a domain of 2^20 block layers: the same bits as
    at the bottom of a low one, and a first call's host work that follows the
    blocks, not the layers between them and below them (a fraction of a
    millisecond; 98 ms with an item list walked layer by layer)."""
    bsx, low, tall = 8, 24, 1 << 20
    r = np.random.default_rng(7)
    layers = np.array([4, 5, 6, 9, 17, 18])
    values = r.uniform(0, 1, (len(layers), bsx ** 3)).astype(np.float32)
    params = msbg.PdeParams(0.05, 10, False)
    got, took = [], []
    for height, up in ((low, 0), (tall, tall - low)):
        g = msbg.SparseGrid(ctx, bsx, bsx, bsx * height, 0.25, 0.75, bsx)
        ids = (layers + up).astype(np.uint64)
        g.write_blocks(ids, values)
        sw = msbg.Sweeper(g)
        ctx.synchronize()
        for turn in range(3):  # another active set each time: another plan
            active = ids if turn == 0 else ids[turn:]
            t0 = time.perf_counter()
            sw.sweep(active, 0, params)
            ctx.synchronize()
            took.append(time.perf_counter() - t0)
        got.append(g.read_blocks(ids))
        if not up:  # a gap of a million layers between two blocks as well
            g2 = msbg.SparseGrid(ctx, bsx, bsx, bsx * tall, 0.25, 0.75, bsx)
            far = np.array([4, 5, 6, tall - low + 9, tall - low + 17, tall - low + 18], np.uint64)
            g2.write_blocks(far, values)
            for turn in range(3):
                msbg.Sweeper(g2).sweep(far if turn == 0 else far[turn:], 0, params)
            got.append(g2.read_blocks(far))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    assert min(took[3:]) < 0.03, took
