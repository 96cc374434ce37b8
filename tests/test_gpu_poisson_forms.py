"""Pressure solves at the sizes where a kernel's form changes: the restriction
with four lanes a coarse cell or with one thread (200,000 coarse cells), the
quad tile with 4 or 16 planes a CTA (2,048 blocks of 16^3), CG's dot products
inside its kernels or as kernels of their own (8,192 of its partial sums), and the
last smoothing sweep ending in either buffer.  Checked by the residual in FP64,
the oracle's iteration count where it is quick, and the bits of a second solve."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def some_blocks(nb, count, seed):
    return np.sort(np.random.default_rng(seed).permutation(nb ** 3)[:count])


def solve_twice(msbg, ctx, oracle, act, nb, bsx, method, mode, nu=(2, 2), oracle_below=600000):
    s = nb * bsx
    P = msbg.Poisson(ctx, s, s, s, bsx, act)
    P.set_smoother(*nu)
    b = np.random.default_rng(nb + bsx).uniform(-1, 1, P.n).astype(np.float32)
    d_b = torch.from_numpy(b).cuda()
    x = [torch.zeros(P.n, dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()  # the solver has its own stream
    for q in x:
        it, rel, _ = P.solve_device(q, d_b, method=method, tol=1e-6, max_iter=100)
        assert rel <= 1e-6
    assert torch.equal(x[0], x[1])
    ax = oracle.poisson_matvec(act.astype(np.int64), nb, nb, nb, bsx, x[0].cpu().numpy())
    assert np.linalg.norm(b - ax) <= 1.1e-6 * np.linalg.norm(b)
    if P.n <= oracle_below:
        _, h = oracle.poisson_solve(act.astype(np.int64), nb, nb, nb, bsx, b.astype(np.float64), mode=mode, tol=1e-6,
                                    max_iter=100, nu1=nu[0], nu2=nu[1])
        assert abs(it - len(h)) <= 1


@pytest.mark.parametrize("nb,bsx,count", [(4, 32, 48), (4, 32, 49), (6, 32, 200)])
@pytest.mark.parametrize("mode", [0, 1])
def test_restriction_of_the_finest_level(msbg, ctx, oracle, nb, bsx, count, mode):
    """196,608, 200,704 and 819,200 coarse cells under the finest level."""
    solve_twice(msbg, ctx, oracle, some_blocks(nb, count, count), nb, bsx, [msbg.MG, msbg.PCG][mode], mode)


@pytest.mark.parametrize("nb,count", [(13, 2048), (13, 2049), (21, 8192), (21, 8193)])
def test_tiles_and_dot_products_of_large_sets(msbg, ctx, oracle, nb, count):
    """16^3 blocks on both sides of the quad tile's split and of the limit of
    the dot products formed inside the kernels."""
    solve_twice(msbg, ctx, oracle, some_blocks(nb, count, count), nb, 16, msbg.PCG, 1)


SETS = [(1, 16, 1), (5, 16, 60), (9, 8, 300), (13, 16, 2049)]


# (plain cycles diverge on the last set, in the FP64 oracle as well: it is left to CG)
@pytest.mark.parametrize("nu,nb,bsx,count", [(nu, *q) for nu in [(1, 1), (2, 2), (3, 3)] for q in SETS] +
                         [((1, 3), *q) for q in SETS[:3]])
def test_smoother_counts(msbg, ctx, oracle, nu, nb, bsx, count):
    """CG with odd and even sweep counts; with different counts before and
    after, the cycle's post-sweeps end in the other buffer (plain cycles)."""
    mode = 1 if nu[0] == nu[1] else 0
    solve_twice(msbg, ctx, oracle, some_blocks(nb, count, nb), nb, bsx, [msbg.MG, msbg.PCG][mode], mode, nu)
