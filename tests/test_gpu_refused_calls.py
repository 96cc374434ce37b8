"""A call that is refused with a CUDA error leaves nothing behind: the next
calls on the context run."""
import numpy as np
import pytest

from test_gpu_grid import random_sparse
from test_gpu_sweep import assert_same_blocks, run_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stencil", [0, 1])
def test_after_a_sweep_too_large_for_shared_memory(msbg, ctx, oracle, stencil):
    """f32 sweeps of 32^3 blocks with one-cell halos want more shared memory
    than a CTA has."""
    host = random_sparse(msbg, 64, 64, 64, 32, 1.1, 3)
    dev = msbg.SparseGrid.from_host(ctx, host)
    with pytest.raises(msbg.MsbgError):
        msbg.Sweeper(dev).sweep(sorted(host.blocks), stencil, msbg.PdeParams(0.05, 1, False))
    small = random_sparse(msbg, 32, 32, 32, 8, 0.7, 4)
    got = run_device(msbg, ctx, small, sorted(small.blocks), stencil, 0.05, 2, False)
    oracle.sweep(small, sorted(small.blocks), stencil, 0.05, 2, False)
    assert_same_blocks(got, small, np.arange(small.n_blocks))
    assert_same_blocks(dev, host, np.arange(host.n_blocks))
