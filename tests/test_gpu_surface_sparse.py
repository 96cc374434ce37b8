"""The surface splat on blocks of few particles and of many: each width of
CTA and both window pitches, bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_surface import splat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["u16", "f32"])
@pytest.mark.parametrize("bsx,r_particle,nb_dist", [(8, 0.5, 0.25), (8, 3.0, 2.0), (16, 1.0, 1.0), (16, 4.0, 2.5)])
@pytest.mark.parametrize("per_block", [1, 15, 16, 31, 32, 63, 64, 255, 256])
def test_particles_per_block(msbg, ctx, oracle, dtype, bsx, r_particle, nb_dist, per_block):
    r = np.random.default_rng(per_block + bsx)
    s, nb = 3 * bsx, 27
    b = np.arange(nb)
    origin = np.stack([b % 3, b // 3 % 3, b // 9], 1) * bsx
    # the same count in each block, some on cell faces and centres
    pts = np.repeat(origin, per_block, axis=0) + r.uniform(0, bsx, (nb * per_block, 3))
    pts[::5] = np.floor(pts[::5]) + r.choice([0.0, 0.5], (len(pts[::5]), 3))
    pts = np.minimum(pts.astype(np.float32), np.float32(s) - np.float32(1e-3))
    pts = pts[r.permutation(len(pts))]
    g, act, cfg = splat(msbg, ctx, pts, s, dtype, bsx, r_particle, nb_dist)
    want_act = oracle.surface_active(pts, s, s, s, bsx, r_particle + nb_dist)
    assert np.array_equal(act.astype(np.int64), want_act)
    assert np.array_equal(g.read_blocks(act), oracle.density_splat(pts, s, s, s, bsx, r_particle, nb_dist, dtype, want_act))
