"""Sweeps over blocks at the domain's faces, where the halo follows the Neumann
rule (solver.rs:205-209): domains that end at a block face (the halo mirrors
whole planes), domains that cut their last blocks after one, two or more
cells, and domains of a single block layer, where both sides mirror.  Bit
for bit against the oracle: the staging only copies."""
import numpy as np
import pytest

from test_gpu_grid import random_sparse
from test_gpu_sweep import assert_same_blocks, run_device

pytestmark = pytest.mark.gpu

DOMAINS = [
    # sx, sy, sz, bsx
    (16, 16, 16, 16),
    (32, 16, 48, 16),
    (17, 34, 47, 16),
    (64, 30, 33, 32),
    (33, 40, 16, 8),
    (9, 8, 26, 8),
    (12, 9, 4, 4),
]


@pytest.mark.parametrize("domain", DOMAINS)
@pytest.mark.parametrize("stencil", [0, 1, 2])
@pytest.mark.parametrize("dtype", ["f32", "u16", "bf16"])
def test_edge_blocks_match_oracle(msbg, ctx, oracle, domain, stencil, dtype):
    sx, sy, sz, bsx = domain
    if bsx == 32 and dtype == "f32" and stencil != 2:
        pytest.skip("two f32 staging buffers of 32^3 blocks exceed shared memory: the call is refused")
    host = random_sparse(msbg, sx, sy, sz, bsx, 0.8, 11 + stencil, empty=0.1, full=0.9, dtype=dtype)
    for b in range(0, host.n_blocks, 3):  # never an empty set
        host.full.discard(b)
        host.ensure_block(b)
    if dtype == "u16":
        for b in host.blocks:
            host.blocks[b][:] = np.random.default_rng(b).integers(0, 65536, host.N)
    active = list(host.blocks)
    dev = run_device(msbg, ctx, host, active, stencil, 0.05, 3, dtype == "u16")
    oracle.sweep(host, active, stencil, 0.05, 3, dtype == "u16")
    assert_same_blocks(dev, host, np.arange(host.n_blocks))


@pytest.mark.parametrize("extent", [(32, 48, 16), (64, 48, 80)])
@pytest.mark.parametrize("stencil", [0, 1])
def test_multires_edge_blocks_match_oracle(msbg, ctx, oracle, extent, stencil):
    """Mirrored planes of coarse neighbours (multires/halo.rs:187-358)."""
    sx, sy, sz = extent
    fine = msbg.HostGrid("fine", sx, sy, sz, 0.0, 0.0, 16)
    coarse = msbg.HostGrid("coarse", sx // 2, sy // 2, sz // 2, 0.0, 0.0, 8)
    r = np.random.default_rng(sum(extent))
    levels = (r.random(fine.n_blocks) < 0.4).astype(np.uint8)
    for b in range(fine.n_blocks):
        g, cells = (fine, 4096) if levels[b] == 0 else (coarse, 512)
        g.ensure_block(b)
        g.blocks[b][:] = r.uniform(0, 1, cells)
    active = [b for b in range(fine.n_blocks) if levels[b] == 0]
    dfine, dcoarse = msbg.SparseGrid.from_host(ctx, fine), msbg.SparseGrid.from_host(ctx, coarse)
    msbg.Sweeper(dfine).sweep_multires(dcoarse, levels, active, stencil, msbg.PdeParams(0.05, 3, False))
    ctx.synchronize()
    oracle.sweep_multires(fine, coarse, levels, active, stencil, 0.05, 3, False)
    assert_same_blocks(dfine, fine, active)


@pytest.mark.parametrize("iterations", [1, 2, 11])
@pytest.mark.parametrize("stencil", [0, 1])
@pytest.mark.parametrize("extent,keep", [((64, 64, 64), 0.7), ((256, 256, 192), 0.02)])
def test_active_lists_in_any_order(msbg, ctx, oracle, extent, keep, stencil, iterations):
    """Active lists with repeats, absent and constant blocks, in no order, on
    grids that are mostly active (codes from an array) and mostly empty (codes
    from the block map); one, few and many sweeps in a launch."""
    sx, sy, sz = extent
    host = random_sparse(msbg, sx, sy, sz, 8, keep, 5 + stencil, empty=0.1, full=0.9)
    r = np.random.default_rng(sx + iterations)
    active = list(host.blocks) + list(host.full)[:20] + list(r.integers(0, host.n_blocks, 30)) + list(host.blocks)[::3]
    r.shuffle(active)
    active = [int(b) for b in active]
    dev = run_device(msbg, ctx, host, active, stencil, 0.05, iterations, False)
    oracle.sweep(host, active, stencil, 0.05, iterations, False)
    assert_same_blocks(dev, host, np.arange(host.n_blocks))
