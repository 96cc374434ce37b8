"""Sweeps of 16^3 blocks in each of the phase kernel's launch forms (1,024
threads up to 148 blocks a phase, 512 up to 296, 256 beyond), for every
storage type and stencil that takes them; and f32 sweeps on both sides of the
limits between one launch, a cluster per block and pairs of columns.  Bit for bit
against the oracle."""
import numpy as np
import pytest

from test_gpu_grid import random_sparse
from test_gpu_sweep import assert_same_blocks, run_device

pytestmark = pytest.mark.gpu


def phase_grid(msbg, dims, counts, dtype, seed):
    """counts[c] active blocks of colour c in a dims domain."""
    host = random_sparse(msbg, *dims, 16, 0.0, seed, n_full=0, empty=0.1, full=0.9, dtype=dtype)
    full = random_sparse(msbg, 16, 16, 16, 16, 1.1, seed, n_full=0, dtype=dtype).blocks[0]
    r = np.random.default_rng(seed)
    b = np.arange(host.n_blocks)
    x, y, z = b % host.nx, b // host.nx % host.ny, b // (host.nx * host.ny)
    colour = (x & 1) | ((y & 1) << 1) | ((z & 1) << 2)
    active = []
    for c in range(8):
        ids = b[colour == c]
        assert len(ids) >= counts[c]
        active += list(r.permutation(ids)[: counts[c]])
    for i in sorted(active):
        host.ensure_block(int(i))
        host.blocks[int(i)][:] = np.roll(full, int(r.integers(4096)))
    return host, sorted(int(i) for i in active)


# phases on both sides of both limits within one sweep
COUNTS = {"small": [148, 149, 100, 296, 297, 180, 1, 0], "large": [297, 310, 296, 320, 149, 300, 312, 299]}


@pytest.mark.parametrize("counts", ["small", "large"])
@pytest.mark.parametrize("dtype,stencil", [(t, s) for t in ("u16", "bf16", "f16") for s in (0, 1, 2)] + [("f32", 2)])
def test_phase_forms(msbg, ctx, oracle, dtype, stencil, counts):
    host, active = phase_grid(msbg, (224, 224, 224), COUNTS[counts], dtype, 3 + stencil)
    clamp = dtype == "u16"
    dev = run_device(msbg, ctx, host, active, stencil, 0.05 if stencil != 2 else 0.01, 2, clamp)
    oracle.sweep(host, active, stencil, 0.05 if stencil != 2 else 0.01, 2, clamp, threads=oracle.num_threads())
    assert_same_blocks(dev, host, np.array(active))


@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("stencil", [0, 1, 2])
def test_phase_forms_density8(msbg, ctx, oracle, stencil, lanes):
    """The store's generator is indexed by cell, whatever the form."""
    for counts in COUNTS.values():
        host, active = phase_grid(msbg, (224, 224, 224), counts, "u8", 3 + stencil)
        dev = msbg.SparseGrid.from_host(ctx, host)
        sw = msbg.Sweeper(dev, seed=0x2468ACE1, lanes=lanes)
        sw.sweep(active, stencil, msbg.PdeParams(0.05, 1, True))
        pos = oracle.sweep_stochastic(host, active, stencil, 0.05, 1, True, 0x2468ACE1, lanes, 0)
        assert sw.stream_pos == pos
        assert_same_blocks(dev, host, np.array(active))


@pytest.mark.parametrize("dims,counts,stencil", [
    # the 19-tap stencil: clusters up to 296 blocks a phase, single columns above, pairs from 1,184 blocks
    ((320, 320, 320), [296, 297, 400, 60, 148, 1000, 1, 297], 1),
    # (phases of at most 444 blocks let the next one in late)
    ((320, 320, 320), [444, 445, 443, 446, 300, 592, 593, 444], 1),
    ((352, 352, 352), [1184, 1183, 1200, 1100, 1050, 1185, 1000, 1180], 1),
    # the 7-tap stencil: one launch up to 16,384 blocks, a kernel per phase above
    ((416, 416, 416), [2048] * 8, 0),
    ((416, 416, 416), [2048] * 7 + [2049], 0),
])
def test_f32_forms(msbg, ctx, oracle, dims, counts, stencil):
    host, active = phase_grid(msbg, dims, counts, "f32", 9)
    dev = run_device(msbg, ctx, host, active, stencil, 0.05, 2, False)
    oracle.sweep(host, active, stencil, 0.05, 2, False, threads=oracle.num_threads())
    assert_same_blocks(dev, host, np.array(active))
