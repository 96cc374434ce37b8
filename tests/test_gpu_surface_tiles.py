"""The surface splat's tiling against the oracle: footprints of 8 and 9 voxels
(positions on half cells), one particle, many particles in few blocks (their
particles are split over CTAs), windows of several row pitches."""
import numpy as np
import pytest

from test_gpu_surface import splat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["u16", "f32"])
@pytest.mark.parametrize("s,bsx,r_particle,nb_dist,n", [
    (16, 16, 2.0, 2.0, 1),
    (16, 16, 2.0, 2.0, 40000),   # one block, many parts
    (32, 8, 1.0, 0.5, 30000),
    (48, 16, 3.0, 5.5, 5000),    # W = 34
    (64, 32, 1.0, 0.0, 20001),
])
def test_splat_tiles_match_oracle(msbg, ctx, oracle, dtype, s, bsx, r_particle, nb_dist, n):
    r = np.random.default_rng(n + bsx)
    pts = r.uniform(0, s, (n, 3))
    half = n // 3
    pts[:half] = r.integers(0, s, (half, 3)) + r.choice([0.0, 0.5], (half, 3))
    pts = np.minimum(pts.astype(np.float32), np.float32(s) - np.float32(1e-3))
    g, act, cfg = splat(msbg, ctx, pts, s, dtype, bsx, r_particle, nb_dist)
    want_act = oracle.surface_active(pts, s, s, s, bsx, r_particle + nb_dist)
    assert np.array_equal(act.astype(np.int64), want_act)
    want = oracle.density_splat(pts, s, s, s, bsx, r_particle, nb_dist, dtype, want_act)
    assert np.array_equal(g.read_blocks(act), want)
