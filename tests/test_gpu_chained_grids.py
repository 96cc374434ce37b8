"""Chained launches whose grids are too large for an early trigger (more than
4,096 CTAs), among those that are small enough: sweeps of many small blocks bit
for bit against the oracle, and pressure solves whose transfer kernels run one
CTA per block."""
import numpy as np
import pytest
import torch

from test_gpu_grid import random_sparse
from test_gpu_sweep import assert_same_blocks, run_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,stencil", [("u16", 0), ("f32", 2), ("bf16", 1)])
def test_sweeps_of_many_small_blocks(msbg, ctx, oracle, dtype, stencil):
    """About 4,000 blocks in each of seven colours and 5,832 in the last: phases
    on both sides of the limit."""
    host = random_sparse(msbg, 144, 144, 144, 4, 0.69, 5 + stencil, empty=0.1, full=0.9, dtype=dtype)
    n = host.nx
    for b in range(host.n_blocks):  # every block of colour 7
        x, y, z = b % n, b // n % n, b // (n * n)
        if x & y & z & 1:
            host.full.discard(b)
            host.ensure_block(b)
    active = sorted(host.blocks)
    x, y, z = (np.array(active) // d % n for d in (1, n, n * n))
    phases = np.bincount((x & 1) | ((y & 1) << 1) | ((z & 1) << 2), minlength=8)
    assert phases.min() <= 4096 < phases.max()
    dev = run_device(msbg, ctx, host, active, stencil, 0.02, 2, dtype == "u16")
    oracle.sweep(host, active, stencil, 0.02, 2, dtype == "u16", threads=oracle.num_threads())
    assert_same_blocks(dev, host, np.array(active))


@pytest.mark.parametrize("nb,bsx,fraction", [(20, 4, 0.511), (28, 4, 0.4), (20, 8, 0.6)])
def test_solves_of_many_small_blocks(msbg, ctx, oracle, nb, bsx, fraction):
    """4,088 to 8,780 blocks, a CTA each in the transfers."""
    act = np.sort(np.random.default_rng(nb).permutation(nb ** 3)[: int(fraction * nb ** 3)])
    s = nb * bsx
    P = msbg.Poisson(ctx, s, s, s, bsx, act)
    b = np.random.default_rng(bsx).uniform(-1, 1, P.n).astype(np.float32)
    d_b = torch.from_numpy(b).cuda()
    x = [torch.zeros(P.n, dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for q in x:
        it, rel, _ = P.solve_device(q, d_b, method=msbg.PCG, tol=1e-6, max_iter=100)
        assert rel <= 1e-6
    assert torch.equal(x[0], x[1])
    ax = oracle.poisson_matvec(act.astype(np.int64), nb, nb, nb, bsx, x[0].cpu().numpy())
    assert np.linalg.norm(b - ax) <= 1.1e-6 * np.linalg.norm(b)
    if P.n <= 600000:
        _, h = oracle.poisson_solve(act.astype(np.int64), nb, nb, nb, bsx, b.astype(np.float64), mode=1, tol=1e-6, max_iter=100)
        assert abs(it - len(h)) <= 1
