"""CG's dot products formed inside its kernels and the quad tile's z-split,
over hierarchies of other shapes than the shells: block sizes 2 to 32, one
block to thousands, smoother counts odd and even.  The hierarchy and the
algorithm are the oracle's, so iteration counts agree within one and the
solutions within the tolerance of the solve."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def blocks(nb, fraction, seed):
    r = np.random.default_rng(seed)
    return np.sort(r.permutation(nb ** 3)[: max(1, int(fraction * nb ** 3))])


@pytest.mark.parametrize("nu", [(2, 2), (3, 1), (2, 0)])
@pytest.mark.parametrize("nb,bsx,fraction", [
    (1, 16, 1.0),     # 4096 cells: two levels
    (5, 16, 0.5),
    (9, 8, 0.4),
    (20, 4, 0.3),
    (16, 2, 1.0),
    (3, 32, 0.7),
    (12, 16, 1.0),
])
def test_solves_follow_the_oracle(msbg, ctx, oracle, nb, bsx, fraction, nu):
    act = blocks(nb, fraction, nb + bsx)
    s = nb * bsx
    P = msbg.Poisson(ctx, s, s, s, bsx, act)
    P.set_smoother(*nu)
    b = np.random.default_rng(bsx).uniform(-1, 1, P.n).astype(np.float32)
    methods = [(0, msbg.MG)] + ([(1, msbg.PCG)] if nu[0] == nu[1] else [])  # CG wants the symmetric cycle
    for mode, method in methods:
        x = torch.zeros(P.n, dtype=torch.float64, device="cuda")
        d_b = torch.from_numpy(b).cuda()
        torch.cuda.synchronize()  # the solver has its own stream
        it, rel, hist = P.solve_device(x, d_b, method=method, tol=1e-6, max_iter=100)
        assert rel <= 1e-6
        ax = oracle.poisson_matvec(act.astype(np.int64), nb, nb, nb, bsx, x.cpu().numpy())
        assert np.linalg.norm(b - ax) <= 1.1e-6 * np.linalg.norm(b)
        if P.n <= 600000:
            _, h = oracle.poisson_solve(act.astype(np.int64), nb, nb, nb, bsx, b.astype(np.float64), mode=mode, tol=1e-6,
                                        max_iter=100, nu1=nu[0], nu2=nu[1])
            assert abs(it - len(h)) <= 1
        # a second right-hand side in another buffer, then the first again: the same solution
        x2, b2, again = torch.zeros_like(x), torch.flip(d_b, [0]).contiguous(), torch.zeros_like(x)
        torch.cuda.synchronize()
        P.solve_device(x2, b2, method=method, tol=1e-6, max_iter=100)
        assert P.solve_device(again, d_b, method=method, tol=1e-6, max_iter=100)[0] == it
        assert torch.equal(again, x)
