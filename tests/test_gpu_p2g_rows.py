"""The general P2G splat over radii, at the positions where the rows and
faces of a footprint change (cell centres, face planes, their neighbours in
f32) and with cells that hold more particles than a warp stages at once:
every face within one ulp of the FP64 sum of the reference's f32 terms, and
the momentum within the rounding of the stored mass and velocity.  (The
reference's own f32 sums are no yardstick here: over the 400 particles of one
cell they are off by more than their usual 1e-6.)"""
import numpy as np
import pytest

from test_gpu_particles import EPS, device_channels, ulp_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsx", [8, 16])
@pytest.mark.parametrize("r_p", [0.4, 0.5, 1.0, 1.25, 1.5, 1.75, 2.0, 2.5, 3.0])
def test_p2g_rows(msbg, ctx, oracle, r_p, bsx):
    r = np.random.default_rng(int(100 * r_p) + bsx)
    f = np.float32
    edges = np.array([0.0, 0.25, 0.5, 0.75, np.nextafter(f(0.5), f(0)), np.nextafter(f(0.5), f(1)), 0.9999], f)
    base = r.integers(0, 31, (1500, 3)).astype(f) + r.choice(edges, (1500, 3))
    free = r.uniform(0, 31.99, (4000, 3)).astype(f)
    dense = f([9, 9, 9]) + r.uniform(0, 1, (400, 3)).astype(f)
    pos = np.concatenate([base, free, dense]).astype(f)
    vel = r.normal(size=pos.shape).astype(f)
    mass = r.uniform(0.5, 1.5, len(pos)).astype(f)
    mac = msbg.MacGrid(ctx, 32, 32, 32, bsx)
    msbg.particles_to_grid(mac, pos, vel, mass, r_p)
    act = mac.active_blocks()
    want_act = oracle.active_blocks(pos, 32, 32, 32, bsx, r_p)
    assert np.array_equal(act.astype(np.int64), want_act)
    got = device_channels(mac, act)
    terms = oracle.p2g_terms_f64(pos, vel, mass, 32, 32, 32, bsx, r_p, want_act)
    _, absum = oracle.p2g_f64(pos, vel, mass, 32, 32, 32, bsx, r_p, want_act)
    for a in range(3):
        assert ulp_diff(got[a], terms[a].astype(f)).max() <= 1.0
        momentum = got[3 + a].astype(np.float64) * got[a].astype(np.float64)
        assert np.all(np.abs(momentum - terms[3 + a]) <= 4 * EPS * absum[3 + a] + 1e-30)


@pytest.mark.parametrize("bsx", [8, 16])
@pytest.mark.parametrize("n", [1023, 2048, 5000, 70001, 150000])
def test_p2g_uneven_blocks(msbg, ctx, oracle, n, bsx):
    """One block with nearly all particles beside blocks with a single one:
    the kernels that share a block's particles among several CTAs get whole,
    partial and empty shares.  Mass to one ulp of the FP64 sum."""
    r = np.random.default_rng(n + bsx)
    f = np.float32
    lone = f([[20.5, 3.25, 3.5], [31.5, 31.25, 31.75], [0.25, 20.5, 17.0]])
    pos = np.concatenate([r.uniform(bsx, 2 * bsx - 0.01, (n - 3, 3)).astype(f), lone]).astype(f)
    vel = r.normal(size=pos.shape).astype(f)
    mass = r.uniform(0.5, 1.5, n).astype(f)
    mac = msbg.MacGrid(ctx, 32, 32, 32, bsx)
    msbg.particles_to_grid(mac, pos, vel, mass, 1.5)
    act = mac.active_blocks()
    want_act = oracle.active_blocks(pos, 32, 32, 32, bsx, 1.5)
    assert np.array_equal(act.astype(np.int64), want_act)
    got = device_channels(mac, act)
    terms = oracle.p2g_terms_f64(pos, vel, mass, 32, 32, 32, bsx, 1.5, want_act)
    for a in range(3):
        assert ulp_diff(got[a], terms[a].astype(f)).max() <= 1.0
