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
