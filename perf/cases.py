"""Performance cases of the sparse-grid hot path on one B200.

Each case is one pass through the package's entry points (or the C ABI they
bind), with the shapes of the benchmark configurations or of the same ranges:

  flip     one FLIP transfer step on the device: Morton sort, permute, P2G,
           2^3 downsample, multires 19-tap sweeps of the x-face mass, G2P with
           the FLIP/PIC blend
  p2g      particles_to_grid on particles in the caller's order, any radius
  smooth   Sweeper.sweep over a spherical shell of blocks (7, 19 or 25 taps,
           every storage type)
  surface  min-splat of a particle cloud, finalize, clamped 19-tap smoothing
  poisson  a pressure solve from zero to a relative residual of 1e-6
  batch    many uneven pressure solves to 1e-8 in one launch
  conv     one 3x3x3 block-sparse convolution layer of the learned
           preconditioner: forward, data gradient, weight gradient

`listed()` holds fixed cases, `draw(rng)` gives others of the same ranges,
`prepare` makes what a program holds before the call, `run` is one pass,
`work` the bytes and operations a pass cannot do without, and `exact` the
same outputs in 64-bit arithmetic, from torch alone.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STENCILS = {7: 0, 19: 1, 25: 2}
ELEM_BYTES = {"f32": 4, "u16": 2, "bf16": 2, "f16": 2, "u8": 1}
DT, ALPHA = 0.025, 0.95
SWEEPS = 10  # sweeps of the FLIP step's smoother

_shared = {}


def _package():
    """The package (its directory name has a hyphen, so it is loaded by path)."""
    if "msbg_rs_b200" not in sys.modules:
        pkg = os.path.join(ROOT, "msbg-rs_b200")
        spec = importlib.util.spec_from_file_location("msbg_rs_b200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["msbg_rs_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["msbg_rs_b200"]


def _context():
    """One context for the process, as a program on one GPU keeps."""
    if "ctx" not in _shared:
        ctx = _package().Context(0)
        _shared["ctx"] = ctx
        _shared["stream"] = torch.cuda.ExternalStream(ctx.stream(), device=torch.device("cuda", 0))
    return _shared["ctx"], _shared["stream"]


# ---- the cases -------------------------------------------------------------------
def listed():
    return [
        # a small simulation's step: launches, host round trips and latency count
        {"name": "flip_64", "kind": "flip", "size": 64, "ppc": 8},
        # the headline FLIP transfer: 25.4 M particles in 776 level-0 blocks
        {"name": "flip_256", "kind": "flip", "size": 256, "ppc": 8},
        # transfer alone with a narrower kernel, 8^3 blocks, unsorted particles
        {"name": "p2g_r1.5_136", "kind": "p2g", "size": 136, "bsx": 8, "r_p": 1.5, "ppc": 8},
        # the small smoother configuration: 10 sweeps of the 128^3 shell
        {"name": "smooth7_f32_128", "kind": "smooth", "size": 128, "taps": 7, "dtype": "f32", "iterations": 10,
         "thickness": 12, "clamp": False},
        # the smoother on a grid larger than L2 (56,056 blocks, 918 MB)
        {"name": "smooth7_f32_2048", "kind": "smooth", "size": 2048, "taps": 7, "dtype": "f32", "iterations": 10,
         "thickness": 12, "clamp": False},
        # density smoothing of a reconstructed surface, u16 storage, clamped
        {"name": "smooth19_u16_512", "kind": "smooth", "size": 512, "taps": 19, "dtype": "u16", "iterations": 5,
         "thickness": 24, "clamp": True},
        # the phase-field smoother: 25 taps on bf16 storage at 512^3
        {"name": "smooth25_bf16_512", "kind": "smooth", "size": 512, "taps": 25, "dtype": "bf16", "iterations": 10,
         "thickness": 24, "clamp": False},
        # surface reconstruction of a particle cloud (splat, finalize, 5 sweeps)
        {"name": "surface_u16_256", "kind": "surface", "size": 256, "n": 2000003, "dtype": "u16", "r_particle": 2.0,
         "nb_dist": 2.0, "iterations": 5},
        # the pressure solve of the 256^3 layout (3.18 M unknowns)
        {"name": "poisson_256", "kind": "poisson", "size": 256, "bsx": 16, "method": "pcg"},
        # uneven pressure solves of many small domains together
        {"name": "batch_16", "kind": "batch", "problems": 16, "max_edge": 128},
        # the learned preconditioner's middle and coarse layers, one training step of each
        {"name": "conv_32_32_8", "kind": "conv", "size": 256, "lg": 3, "cin": 32, "cout": 32},
        {"name": "conv_64_64_4", "kind": "conv", "size": 256, "lg": 2, "cin": 64, "cout": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flip", "flip", "p2g", "smooth", "smooth", "smooth", "surface", "poisson", "batch", "conv"])
    if kind == "flip":
        return {"kind": kind, "size": 16 * _log_int(rng, 2, 16), "ppc": rng.randint(1, 8)}
    if kind == "p2g":
        bsx = rng.choice([8, 16])
        return {"kind": kind, "size": bsx * _log_int(rng, 32 // bsx, 136 // bsx), "bsx": bsx,
                "r_p": rng.choice([1.0, 1.25, 1.5, 2.0, 2.5, 3.0]), "ppc": rng.randint(2, 8)}
    if kind == "smooth":
        taps = rng.choice([7, 19, 25])
        dtype = rng.choice(["f32", "f32", "u16", "bf16", "f16", "u8"])
        # the largest grids are smoothed with the 7-tap stencil; the wide ones stay at 512
        size = _log_int(rng, 64, 2048 if taps == 7 else 512)
        return {"kind": kind, "size": size, "taps": taps, "dtype": dtype, "iterations": rng.randint(1, 10),
                "thickness": rng.randint(8, 12) if size > 512 else rng.randint(8, 24), "clamp": dtype in ("u16", "u8")}
    if kind == "surface":
        return {"kind": kind, "size": 16 * _log_int(rng, 4, 16), "n": _log_int(rng, 20000, 2000003),
                "dtype": rng.choice(["u16", "u8", "f32"]), "r_particle": rng.choice([1.5, 2.0, 2.5]),
                "nb_dist": rng.choice([1.0, 2.0]), "iterations": rng.randint(1, 5)}
    if kind == "poisson":
        return {"kind": kind, "size": 16 * _log_int(rng, 4, 16), "bsx": rng.choice([8, 16]), "method": rng.choice(["mg", "pcg"])}
    if kind == "batch":
        return {"kind": kind, "problems": rng.randint(2, 16), "max_edge": rng.choice([64, 128])}
    lg = rng.choice([2, 3])
    cin, cout = rng.choice([(16, 32), (32, 32), (32, 16)] if lg == 3 else [(32, 64), (64, 64), (64, 32)])
    return {"kind": "conv", "size": 16 * _log_int(rng, 4, 16), "lg": lg, "cin": cin, "cout": cout}


# ---- geometry and inputs (plain torch and numpy) -------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _band_blocks(nb, bsx, radius, half):
    """Blocks (ids ascending) whose centre is within `half` cells of the sphere
    of `radius` around the domain centre: the level-0 blocks of the FLIP layout."""
    b = torch.arange(nb, device="cuda", dtype=torch.float64)
    c = (b + 0.5) * bsx - nb * bsx / 2
    d = (c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2).sqrt() - radius
    return torch.nonzero((d.abs() < half).reshape(-1)).reshape(-1)


def _levels(nb, bsx, radius):
    b = torch.arange(nb, device="cuda", dtype=torch.float64)
    c = (b + 0.5) * bsx - nb * bsx / 2
    d = ((c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2).sqrt() - radius).abs().reshape(-1)
    return torch.where(d < 16, 0, torch.where(d < 48, 1, 2)).to(torch.uint8).cpu().numpy()


def _shell_blocks(size, thickness, r=None):
    """16^3 blocks of a size^3 domain meeting the shell of radius r (0.35 size)."""
    nb = (size + 15) // 16
    lo = torch.arange(nb, device="cuda", dtype=torch.float64) * 16 - size / 2
    hi = lo + 16
    near = torch.clamp(torch.maximum(lo, -hi), min=0)
    far = torch.maximum(lo.abs(), hi.abs())
    dmin = (near[:, None, None] ** 2 + near[None, :, None] ** 2 + near[None, None, :] ** 2).sqrt()
    dmax = (far[:, None, None] ** 2 + far[None, :, None] ** 2 + far[None, None, :] ** 2).sqrt()
    r = 0.35 * size if r is None else r
    return torch.nonzero(((dmin <= r + thickness / 2) & (dmax >= r - thickness / 2)).reshape(-1)).reshape(-1)


def _block_coords(ids, nb):
    return ids % nb, (ids // nb) % nb, ids // (nb * nb)


def _cell_coords(ids, nb, bsx):
    """Integer coordinates [blocks][bsx^3][3] of every cell, payload order."""
    v = torch.arange(bsx ** 3, device="cuda")
    bx, by, bz = _block_coords(ids, nb)
    return torch.stack([bx[:, None] * bsx + v % bsx, by[:, None] * bsx + (v // bsx) % bsx,
                        bz[:, None] * bsx + v // (bsx * bsx)], -1)


def _particles(case, seed, blocks, nb, bsx):
    """ppc particles per cell of `blocks`, jittered inside the cell, in random order."""
    g = _gen(seed)
    origin = _cell_coords(blocks, nb, bsx).reshape(-1, 3).to(torch.float32).repeat_interleave(case["ppc"], 0)
    pos = origin + torch.rand(origin.shape, generator=g, device="cuda")
    pos = torch.minimum(pos, torch.nextafter(origin + 1, origin))
    pos = pos[torch.randperm(len(pos), generator=g, device="cuda")].contiguous()
    vel = torch.randn(pos.shape, generator=g, device="cuda")
    mass = torch.ones(len(pos), device="cuda")
    return pos, vel, mass


def _smooth_values(case, seed, ids):
    """7 taps: U[-1, 1] (the smoother configuration); 19 and 25 taps: a phase
    profile across the shell with a little noise, in [0, 1]."""
    g = _gen(seed)
    if case["taps"] == 7 and not case["clamp"]:
        return torch.rand((len(ids), 4096), generator=g, device="cuda") * 2 - 1
    size = case["size"]
    nb = (size + 15) // 16
    out = torch.empty((len(ids), 4096), device="cuda")
    for s in range(0, len(ids), 4096):
        c = _cell_coords(ids[s:s + 4096], nb, 16).to(torch.float32) + (0.5 - size / 2)
        phi = c.square().sum(-1).sqrt() - 0.35 * size
        noise = torch.rand(phi.shape, generator=g, device="cuda") - 0.5
        out[s:s + 4096] = (0.5 * (1 - torch.tanh(phi / 4)) + 0.1 * noise).clamp(0, 1)
    return out


def _stored(values, dtype):
    if dtype == "f32":
        return values
    if dtype == "u16":
        return (values.clamp(0, 1) * 65535 + 0.5).floor().to(torch.int32).to(torch.int16)
    if dtype == "u8":
        return (values.clamp(0, 1) * 255 + 0.5).floor().to(torch.uint8)
    return values.to(torch.bfloat16 if dtype == "bf16" else torch.float16)


def _cloud(case, seed):
    """Particles on a bumpy sphere shell, the kind of cloud a surface is built from."""
    g = _gen(seed)
    d = torch.randn((case["n"], 3), generator=g, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    r = case["size"] * (0.3 + 0.03 * torch.sin(6 * d[:, :1]) * torch.cos(5 * d[:, 1:2]))
    r = r + 4 * (torch.rand((case["n"], 1), generator=g, device="cuda") - 0.5)
    return (case["size"] / 2 + r * d).contiguous()


def _smooth_rhs(seed, ids, nb, bsx):
    """Divergence of a random smooth velocity field (32 Gaussian blobs) at the
    cell centres, [cells] f32: the pressure solve's right-hand side."""
    g = _gen(seed)
    x = _cell_coords(ids, nb, bsx).reshape(-1, 3).to(torch.float64) + 0.5
    centre = x[torch.randint(0, len(x), (32,), generator=g, device="cuda")]
    sigma = 4 + 12 * torch.rand(32, generator=g, device="cuda", dtype=torch.float64)
    amp = torch.randn((32, 3), generator=g, device="cuda", dtype=torch.float64)
    out = torch.zeros(len(x), device="cuda", dtype=torch.float64)
    for i in range(32):
        d = x - centre[i]
        out -= (d @ amp[i]) / sigma[i] ** 2 * torch.exp(-d.square().sum(1) / (2 * sigma[i] ** 2))
    return out.to(torch.float32)


def _batch_problems(case, seed):
    """Geometries are the case's own (a program's plan); right-hand sides the seed's."""
    geo = np.random.default_rng(case["problems"] * 1000 + case["max_edge"])
    g = _gen(seed)
    edges = [e for e in (32, 64, 128) if e <= case["max_edge"]]
    out = []
    for p in range(case["problems"]):
        edge = edges[-1] if p == 0 else int(geo.choice(edges))
        bsx = 16 if p == 0 else int(geo.choice([8, 16]))
        nb = edge // bsx
        fraction = geo.uniform(0.05, 0.6)
        b = np.arange(nb)
        bz, by, bx = np.meshgrid(b, b, b, indexing="ij")
        mid = (np.stack([bx, by, bz], -1).reshape(-1, 3) + 0.5) * bsx
        c, r = geo.uniform(0.3, 0.7, 3) * edge, geo.uniform(0.2, 0.45) * edge
        d = np.abs(np.linalg.norm(mid - c, axis=1) - r)
        k = max(1, int(np.ceil(fraction * nb ** 3)))
        ids = np.sort(np.argsort(d, kind="stable")[:k]).astype(np.uint64)
        rhs = torch.rand(k * bsx ** 3, generator=g, device="cuda") * 2 - 1
        out.append((edge, bsx, ids, rhs - rhs.mean()))
    return out


def _conv_inputs(case, seed):
    g = _gen(seed)
    nb = case["size"] // 16
    ids = _band_blocks(nb, 16, 0.35 * case["size"], 16.0)
    cells = len(ids) * 8 ** case["lg"]
    # activations after a ReLU, gradients without one, weights of He scale
    x = torch.randn((cells, case["cin"]), generator=g, device="cuda").clamp(min=0).to(torch.bfloat16)
    dy = torch.randn((cells, case["cout"]), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((27, case["cout"], case["cin"]), generator=g, device="cuda") * math.sqrt(2 / (27 * case["cin"]))).to(torch.bfloat16)
    bias = torch.randn(case["cout"], generator=g, device="cuda") * 0.1
    return ids, _neighbours27(ids, nb), x, dy, w, bias


def _slots(ids, nb, pad):
    """Dense block id -> slot table; `pad` where the block is not in the set."""
    t = torch.full((nb ** 3,), pad, device="cuda", dtype=torch.int64)
    t[ids] = torch.arange(len(ids), device="cuda")
    return t


def _neighbours27(ids, nb):
    """[blocks][27] slot of every neighbour block, -1 where absent."""
    slot = _slots(ids, nb, -1)
    bx, by, bz = _block_coords(ids, nb)
    out = torch.full((len(ids), 27), -1, device="cuda", dtype=torch.int32)
    for t in range(27):
        x, y, z = bx + t % 3 - 1, by + (t // 3) % 3 - 1, bz + t // 9 - 1
        ok = (x >= 0) & (x < nb) & (y >= 0) & (y < nb) & (z >= 0) & (z < nb)
        at = (x + y * nb + z * nb * nb).clamp(0, nb ** 3 - 1)
        out[:, t] = torch.where(ok, slot[at], -1).to(torch.int32)
    return out


class _DeviceArray:
    """A library-owned device buffer as torch sees it (no copy); torch keeps
    this object, and it the buffer's owner, as long as the tensor lives."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": typestr, "version": 3}


def _view(owner, ptr, shape, dtype):
    name = {torch.float32: "<f4", torch.float64: "<f8", torch.int16: "<i2", torch.uint8: "|u1",
            torch.bfloat16: "<i2", torch.float16: "<f2"}[dtype]
    t = torch.as_tensor(_DeviceArray(owner, ptr, shape, name), device="cuda")
    return t.view(torch.bfloat16) if dtype is torch.bfloat16 else t


GRID_TORCH = {"f32": torch.float32, "u16": torch.int16, "bf16": torch.bfloat16, "f16": torch.float16, "u8": torch.uint8}


def _payload(grid, owner):
    ptr, n = grid.payload_device_ptr()
    return _view(owner, ptr, (n, grid.N), GRID_TORCH[grid.dtype])


# ---- prepare -------------------------------------------------------------------------
def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, seed)
    state["case"] = case
    torch.cuda.synchronize()  # the inputs are made on torch's stream, the library has its own
    return state


def _prepare_flip(case, seed):
    M, (ctx, stream) = _package(), _context()
    size, nb = case["size"], case["size"] // 16
    blocks = _band_blocks(nb, 16, 0.35 * size, 16.0)
    pos, vel, mass = _particles(case, seed, blocks, nb, 16)
    n = len(mass)
    mac = M.MacGrid(ctx, size, size, size, 16)
    return {"M": M, "ctx": ctx, "n": n, "pos": pos, "vel": vel, "mass": mass, "mac": mac,
            "coarse": M.SparseGrid(ctx, size // 2, size // 2, size // 2, 0.0, 0.0, 8, name="coarse_mass_x"),
            "levels": _levels(nb, 16, 0.35 * size), "sweeper": M.Sweeper(mac.mass(0)), "sampler": M.MacSampler(mac, M.CLAMP),
            "keys": torch.empty(n, dtype=torch.int64, device="cuda"), "perm": torch.empty(n, dtype=torch.int32, device="cuda"),
            "spos": torch.empty_like(pos), "svel": torch.empty_like(vel), "smass": torch.empty_like(mass),
            "out": torch.empty_like(vel)}


def _prepare_p2g(case, seed):
    M, (ctx, stream) = _package(), _context()
    size, bsx = case["size"], case["bsx"]
    blocks = _band_blocks(size // bsx, bsx, 0.35 * size, 12.0)
    pos, vel, mass = _particles(case, seed, blocks, size // bsx, bsx)
    return {"M": M, "mac": M.MacGrid(ctx, size, size, size, bsx), "pos": pos, "vel": vel, "mass": mass, "n": len(mass)}


def _prepare_smooth(case, seed):
    M, (ctx, stream) = _package(), _context()
    size = case["size"]
    ids = _shell_blocks(size, case["thickness"])
    payload = _stored(_smooth_values(case, seed, ids), case["dtype"]).contiguous()
    active = ids.cpu().numpy().astype(np.uint64)
    torch.cuda.synchronize()
    grid = M.SparseGrid(ctx, size, size, size, 0.0, 1.0, 16, case["dtype"])
    M._lib.call("msbg_grid_write_blocks_device", grid.handle, M._lib.ptr(active), len(active), M._lib.ptr(payload))
    ctx.synchronize()
    return {"M": M, "grid": grid, "active": active, "sweeper": M.Sweeper(grid),
            "params": M.PdeParams(DT, case["iterations"], case["clamp"])}


def _prepare_surface(case, seed):
    M, (ctx, stream) = _package(), _context()
    size = case["size"]
    cfg = M.SurfaceConfig(size, size, size, r_particle=case["r_particle"], nb_dist=case["nb_dist"],
                          n_smooth_iters=case["iterations"], smooth_dt=0.05)
    grid = M.SparseGrid(ctx, size, size, size, 0.0, 1.0, 16, case["dtype"], name="surface")
    # the band the surface moves in is materialised once, as a simulation that
    # rebuilds its surface every frame would have it after the first frames
    reach = 2 * (0.03 * size + 2 + cfg.r_scan + 2)
    grid.ensure_blocks(_shell_blocks(size, reach, 0.3 * size).cpu().numpy())
    return {"M": M, "grid": grid, "cfg": cfg, "pos": _cloud(case, seed)}


def _prepare_poisson(case, seed):
    M, (ctx, stream) = _package(), _context()
    size, bsx = case["size"], case["bsx"]
    ids = _band_blocks(size // bsx, bsx, 0.35 * size, 16.0)
    P = M.Poisson(ctx, size, size, size, bsx, ids.cpu().numpy())
    b = _smooth_rhs(seed, ids, size // bsx, bsx)
    return {"M": M, "P": P, "b": b, "x": torch.empty_like(b), "stream": stream,
            "method": M.PCG if case["method"] == "pcg" else M.MG}


def _prepare_batch(case, seed):
    M, (ctx, stream) = _package(), _context()
    problems = _batch_problems(case, seed)
    batch = M.Batch(ctx, [((e, e, e), bsx, ids) for e, bsx, ids, _ in problems], tune=True)
    for p, (_, _, _, rhs) in enumerate(problems):
        batch.set_rhs(p, rhs.cpu().numpy())
    groups = []
    for g in range(batch.n_groups):
        _, x, cells, _ = batch.buffers(g)
        groups.append((_view(batch, x, (cells,), torch.float64), torch.empty(cells, device="cuda")))
    return {"M": M, "batch": batch, "groups": groups, "stream": stream}


def _prepare_conv(case, seed):
    M, (ctx, stream) = _package(), _context()
    ids, nbr, x, dy, w, bias = _conv_inputs(case, seed)
    return {"M": M, "ctx": ctx, "blocks": len(ids), "nbr": nbr, "x": x, "dy": dy, "w": w, "bias": bias,
            "wt": w.flip(0).transpose(1, 2).contiguous(),  # mirrored taps, transposed: the data gradient's weights
            "y": torch.empty_like(dy), "dx": torch.empty_like(x),
            "dw": torch.empty((27, case["cout"], case["cin"]), device="cuda")}


# ---- run -----------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_flip(s):
    M, ctx, n, mac = s["M"], s["ctx"], s["n"], s["mac"]
    call, ptr = M._lib.call, M._lib.ptr
    call("msbg_morton_sort_device", ctx.handle, ptr(s["pos"]), n, ptr(s["keys"]), ptr(s["perm"]))
    call("msbg_permute_device", ctx.handle, ptr(s["perm"]), n, 3, ptr(s["pos"]), ptr(s["spos"]))
    call("msbg_permute_device", ctx.handle, ptr(s["perm"]), n, 3, ptr(s["vel"]), ptr(s["svel"]))
    call("msbg_permute_device", ctx.handle, ptr(s["perm"]), n, 1, ptr(s["mass"]), ptr(s["smass"]))
    M.particles_to_grid_sorted_device(mac, s["spos"], s["svel"], s["smass"], s["keys"], n, 2.0)
    act = mac.active_blocks()
    fine = act[s["levels"][act.astype(np.int64)] == 0]
    M.downsample_channel_avg(s["coarse"], mac.mass(0))
    s["sweeper"].sweep_multires(s["coarse"], s["levels"], fine, M.Stencil.MeanCurvature, M.PdeParams(DT, SWEEPS, False))
    M.g2p_flip_device(s["sampler"], s["spos"], n, s["svel"], ALPHA, s["out"])
    return {"velocity": s["out"], "positions": s["spos"], "keys": s["keys"], "perm": s["perm"], "mass_x": _payload(mac.mass(0), mac),
            "mass_y": _payload(mac.mass(1), mac)}


def _run_p2g(s):
    s["M"].particles_to_grid_device(s["mac"], s["pos"], s["vel"], s["mass"], s["n"], s["case"]["r_p"])
    return {"mass": [_payload(s["mac"].mass(a), s["mac"]) for a in range(3)], "velocity": [_payload(s["mac"].velocity(a), s["mac"]) for a in range(3)]}


def _run_smooth(s):
    s["sweeper"].sweep(s["active"], s["M"].Stencil(STENCILS[s["case"]["taps"]]), s["params"])
    return _payload(s["grid"], s["grid"])


def _run_surface(s):
    M, cfg = s["M"], s["cfg"]
    act = M.surface.splat_device(s["grid"], s["pos"], len(s["pos"]), cfg)
    M.surface.finalize(s["grid"], act, cfg)
    M.Sweeper(s["grid"]).sweep(act, M.Stencil.MeanCurvature, M.PdeParams(cfg.smooth_dt, cfg.n_smooth_iters, True))
    return _payload(s["grid"], s["grid"])


def _run_poisson(s):
    with torch.cuda.stream(s["stream"]):
        s["x"].zero_()
    s["P"].solve_device(s["x"], s["b"], method=s["method"], tol=1e-6, max_iter=100)
    return s["x"]


def _run_batch(s):
    s["batch"].solve(tol=1e-8, iters_per_cycle=8, max_cycles=60)
    with torch.cuda.stream(s["stream"]):
        for x64, x32 in s["groups"]:  # the pressure as the f32 field a simulation keeps
            x32.copy_(x64)
    return [x32 for _, x32 in s["groups"]]


def _run_conv(s):
    M, c = s["M"], s["case"]
    call, ptr, h, nb = M._lib.call, M._lib.ptr, s["ctx"].handle, s["blocks"]
    call("msbg_conv3_forward_device", h, ptr(s["nbr"]), nb, c["lg"], c["cin"], c["cout"], ptr(s["x"]), ptr(s["w"]), ptr(s["bias"]),
         1, 0, ptr(s["y"]))
    call("msbg_conv3_forward_device", h, ptr(s["nbr"]), nb, c["lg"], c["cout"], c["cin"], ptr(s["dy"]), ptr(s["wt"]), None,
         0, 0, ptr(s["dx"]))
    call("msbg_conv3_wgrad_device", h, ptr(s["nbr"]), nb, c["lg"], c["cin"], c["cout"], ptr(s["x"]), ptr(s["dy"]), ptr(s["dw"]))
    return {"y": s["y"], "dx": s["dx"], "dw": s["dw"]}


# ---- work ----------------------------------------------------------------------------
def _count(size, bsx, half):
    """Number of _band_blocks, without a GPU."""
    nb = size // bsx
    c = (np.arange(nb) + 0.5) * bsx - nb * bsx / 2
    d = np.sqrt(c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2) - 0.35 * size
    return int((np.abs(d) < half).sum())


def _shell_count(size, thickness):
    nb = (size + 15) // 16
    lo = np.arange(nb) * 16.0 - size / 2
    hi = lo + 16
    near, far = np.maximum(np.maximum(lo, -hi), 0) ** 2, np.maximum(np.abs(lo), np.abs(hi)) ** 2
    dmin = np.sqrt(near[:, None, None] + near[None, :, None] + near[None, None, :])
    dmax = np.sqrt(far[:, None, None] + far[None, :, None] + far[None, None, :])
    return int(((dmin <= 0.35 * size + thickness / 2) & (dmax >= 0.35 * size - thickness / 2)).sum())


def work(case):
    kind = case["kind"]
    if kind == "flip":
        blocks = _count(case["size"], 16, 16.0)
        n = blocks * 4096 * case["ppc"]
        # particles in (pos, vel, mass) and new velocities, sorted positions, keys and order out;
        # six face channels written once. Per particle and direction 4^3 faces of about 12
        # operations in P2G; 3 x 21 in G2P
        return {"bytes": n * (28 + 24 + 12) + blocks * 4096 * 24, "flops": n * (3 * 64 * 12 + 63) + blocks * 4096 * 60 * SWEEPS}
    if kind == "p2g":
        blocks = _count(case["size"], case["bsx"], 12.0)
        n = blocks * case["bsx"] ** 3 * case["ppc"]
        faces = (2 * case["r_p"]) ** 3
        return {"bytes": n * 28 + blocks * case["bsx"] ** 3 * 24, "flops": n * 3 * faces * 12}
    if kind == "smooth":
        cells = _shell_count(case["size"], case["thickness"]) * 4096
        return {"bytes": 2 * ELEM_BYTES[case["dtype"]] * cells, "flops": cells * case["iterations"] * {7: 25, 19: 60, 25: 45}[case["taps"]]}
    if kind == "surface":
        r = case["r_particle"] + case["nb_dist"]
        cells = 4 * math.pi * (0.3 * case["size"]) ** 2 * (2 * r + 4)
        return {"bytes": case["n"] * 12 + cells * ELEM_BYTES[case["dtype"]],
                "flops": case["n"] * (4 / 3 * math.pi * r ** 3) * 6 + cells * 60 * case["iterations"]}
    if kind == "poisson":
        cells = _count(case["size"], case["bsx"], 16.0) * case["bsx"] ** 3
        # right-hand side in, solution out; about 12 V(2,2)-cycles of some 80 operations a cell
        return {"bytes": 8 * cells, "flops": cells * 12 * 80}
    if kind == "batch":
        cells = case["problems"] * 0.3 * (case["max_edge"] / 1.6) ** 3
        return {"bytes": 8 * cells, "flops": cells * 16 * 80}
    blocks = _count(case["size"], 16, 16.0)
    cells = blocks * 8 ** case["lg"]
    pair = case["cin"] * case["cout"]
    return {"bytes": cells * 2 * (2 * case["cin"] + 2 * case["cout"]) + 27 * pair * 8, "flops": 3 * 2 * 27 * pair * cells}


# ---- the same in 64 bits ---------------------------------------------------------------
def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


def _splat64(pos, vel, mass, size, r_p):
    """Face masses and momenta as dense [3][size^3] arrays:
    w = max(1 - |face - p|^2 / r_p^2, 0)^3 at the right faces of the cells."""
    m = [torch.zeros(size ** 3, device="cuda", dtype=torch.float64) for _ in range(3)]
    q = [torch.zeros(size ** 3, device="cuda", dtype=torch.float64) for _ in range(3)]
    reach = int(math.ceil(r_p))
    chunk = 1 << 23
    for s in range(0, len(pos), chunk):
        p, v, w0 = pos[s:s + chunk].double(), vel[s:s + chunk].double(), mass[s:s + chunk].double()
        cell = p.floor().long()
        for a in range(3):
            off = torch.full((3,), 0.5, device="cuda", dtype=torch.float64)
            off[a] = 1.0
            d = [[(cell[:, ax] + o) + off[ax] - p[:, ax] for o in range(-reach - 1, reach + 1)] for ax in range(3)]
            for kz in range(2 * reach + 2):
                for ky in range(2 * reach + 2):
                    dyz = d[2][kz].square() + d[1][ky].square()
                    y, z = cell[:, 1] + ky - reach - 1, cell[:, 2] + kz - reach - 1
                    oyz = (y >= 0) & (y < size) & (z >= 0) & (z < size) & (dyz < r_p * r_p)
                    sel = torch.nonzero(oyz).reshape(-1)
                    if not len(sel):
                        continue
                    base, dyz_s, w_s, v_s, c_s = (y * size + z * size * size)[sel], dyz[sel], w0[sel], v[sel, a], cell[sel, 0]
                    for kx in range(2 * reach + 2):
                        x = c_s + kx - reach - 1
                        w = (1 - (d[0][kx][sel].square() + dyz_s) / (r_p * r_p)).clamp(min=0) ** 3 * w_s
                        w = torch.where((x >= 0) & (x < size), w, 0)
                        at = base + x.clamp(0, size - 1)
                        m[a].index_add_(0, at, w)
                        q[a].index_add_(0, at, w * v_s)
    return m, [torch.where(mm > 0, qq / torch.where(mm > 0, mm, 1), 0) for mm, qq in zip(m, q)]


def _p2g_active(pos, size, bsx, r_p):
    """Blocks within r_p + 1 of a particle, ascending (the transfer's block set, in its own f32 rule)."""
    nb = size // bsx
    mark = torch.zeros(nb ** 3, device="cuda", dtype=torch.bool)
    b, r = pos / float(bsx), float(np.float32(r_p + 1.0) / np.float32(bsx))
    lo = (b - r).trunc().long().clamp(min=0)
    hi = (b + r).trunc().long().clamp(max=nb - 1)
    for k in range(8):
        c = [torch.where(torch.tensor(bool(k >> ax & 1), device="cuda"), hi[:, ax], lo[:, ax]) for ax in range(3)]
        mark[c[0] + c[1] * nb + c[2] * nb * nb] = True
    return torch.nonzero(mark).reshape(-1)


def _to_blocks(dense, ids, size, bsx):
    c = _cell_coords(ids, size // bsx, bsx)
    return dense[c[..., 0] + c[..., 1] * size + c[..., 2] * size * size]


def _sample64(field, p, size):
    """Cell-centred trilinear samples (clamped at the domain) of a dense field."""
    f = p.floor()
    t = p - f
    i = f.long()
    out = torch.zeros(len(p), device="cuda", dtype=torch.float64)
    for k in range(8):
        at, w = 0, 1
        for ax in range(3):
            o = k >> ax & 1
            at = at + (i[:, ax] + o).clamp(0, size - 1) * size ** ax
            w = w * (t[:, ax] if o else 1 - t[:, ax])
        out += field[at] * w
    return out


def _spread21(v):
    out = torch.zeros_like(v)
    for k in range(21):
        out |= (v >> k & 1) << (3 * k)
    return out


def _exact_flip(case, seed):
    size, nb = case["size"], case["size"] // 16
    pos, vel, mass = _particles(case, seed, _band_blocks(nb, 16, 0.35 * size, 16.0), nb, 16)
    c = pos.long()
    keys, perm = (_spread21(c[:, 0]) | _spread21(c[:, 1]) << 1 | _spread21(c[:, 2]) << 2).sort(stable=True)
    m, u = _splat64(pos, vel, mass, size, 2.0)
    spos, out = pos[perm], vel[perm].double() * ALPHA
    for a in range(3):
        q = spos.double()
        q[:, a] -= 0.5  # faces sit half a cell to the right of the centres
        out[:, a] += (1 - ALPHA) * _sample64(u[a], q - 0.5, size)
    act = _p2g_active(pos, size, 16, 2.0)
    return {"velocity": out, "positions": spos, "keys": keys, "perm": perm.int(), "mass_x": None, "mass_y": _to_blocks(m[1], act, size, 16)}


def _exact_p2g(case, seed):
    size, bsx = case["size"], case["bsx"]
    pos, vel, mass = _particles(case, seed, _band_blocks(size // bsx, bsx, 0.35 * size, 12.0), size // bsx, bsx)
    m, u = _splat64(pos, vel, mass, size, case["r_p"])
    act = _p2g_active(pos, size, bsx, case["r_p"])
    return {"mass": [_to_blocks(x, act, size, bsx) for x in m], "velocity": [_to_blocks(x, act, size, bsx) for x in u]}


def _exact_smooth(case, seed):
    if case["dtype"] in ("u16", "u8"):
        return None  # whole numbers
    size, taps = case["size"], case["taps"]
    nb, halo = (size + 15) // 16, 2 if taps == 25 else 1
    H = 16 + 2 * halo
    ids = _shell_blocks(size, case["thickness"])
    f = torch.zeros((len(ids) + 1, 4096), device="cuda", dtype=torch.float64)  # last block: what is absent
    f[:-1] = _stored(_smooth_values(case, seed, ids), case["dtype"]).double()
    slot = _slots(ids, nb, len(ids))
    bx, by, bz = _block_coords(ids, nb)
    colour = (bx & 1) | (by & 1) << 1 | (bz & 1) << 2

    def resolve(b):  # [blocks][H] cells of a halo row, mirrored at the domain's faces
        g = (b[:, None] * 16 + torch.arange(-halo, 16 + halo, device="cuda")) % (2 * size)
        return torch.where(g >= size, 2 * size - 1 - g, g)

    for _ in range(case["iterations"]):
        for c in range(8):
            mine = torch.nonzero(colour == c).reshape(-1)
            new = []
            for part in mine.split(2048):
                x, y, z = (resolve(b[part]) for b in (bx, by, bz))
                block = (x >> 4)[:, None, None, :] + ((y >> 4) * nb)[:, None, :, None] + ((z >> 4) * nb * nb)[:, :, None, None]
                vid = (x & 15)[:, None, None, :] + ((y & 15) * 16)[:, None, :, None] + ((z & 15) * 256)[:, :, None, None]
                h = f.view(-1)[slot[block] * 4096 + vid]
                new.append(_stencil64(h, taps, halo, H, case["clamp"]).reshape(len(part), 4096))
            if new:
                f[mine] = torch.cat(new)
    return f[:-1]


def _stencil64(h, taps, halo, H, clamp):
    def at(dx=0, dy=0, dz=0):
        s = [slice(halo + d, H - halo + d) for d in (dz, dy, dx)]
        return h[:, s[0], s[1], s[2]]

    c, xm, xp, ym, yp, zm, zp = at(), at(-1), at(1), at(0, -1), at(0, 1), at(0, 0, -1), at(0, 0, 1)
    fx, fy, fz = (xp - xm) / 2, (yp - ym) / 2, (zp - zm) / 2
    g2 = fx * fx + fy * fy + fz * fz
    faces = xm + xp + ym + yp + zm + zp
    if taps == 7:
        new = c + DT * (faces - 6 * c) * g2.sqrt()
    elif taps == 19:
        fxy = (at(1, 1) - at(1, -1) - at(-1, 1) + at(-1, -1)) / 4
        fxz = (at(1, 0, 1) - at(1, 0, -1) - at(-1, 0, 1) + at(-1, 0, -1)) / 4
        fyz = (at(0, 1, 1) - at(0, 1, -1) - at(0, -1, 1) + at(0, -1, -1)) / 4
        fxx, fyy, fzz = xm + xp - 2 * c, ym + yp - 2 * c, zm + zp - 2 * c
        num = (fy * fy + fz * fz) * fxx + (fx * fx + fz * fz) * fyy + (fx * fx + fy * fy) * fzz - 2 * (fx * fy * fxy + fx * fz * fxz + fy * fz * fyz)
        new = c + (DT * torch.where(g2 > 1e-7, num / torch.where(g2 > 1e-7, g2, 1), 0)).clamp(-0.1, 0.1)
    else:
        far = at(-2) + at(2) + at(0, -2) + at(0, 2) + at(0, 0, -2) + at(0, 0, 2)
        edges = sum(at(i, j) + at(i, 0, j) + at(0, i, j) for i in (-1, 1) for j in (-1, 1))
        new = c + (-DT * (42 * c - 12 * faces + far + 2 * edges) * g2.sqrt()).clamp(-0.1, 0.1)
    return new.clamp(0, 1) if clamp else new


def _solve64(ids, nb, bsx, b):
    """A x = b, A the 7-point operator (6 on the diagonal, zero values outside
    the blocks), by conjugate gradients to a relative residual of 1e-12."""
    cells = len(ids) * bsx ** 3
    slot = _slots(ids, nb + 2, -1)  # unused ids: replaced below by the padded numbering
    bx, by, bz = _block_coords(ids, nb)
    slot = _slots((bx + 1) + (by + 1) * (nb + 2) + (bz + 1) * (nb + 2) ** 2, nb + 2, -1)
    c = _cell_coords(ids, nb, bsx).reshape(-1, 3) + bsx
    near = []
    for ax in range(3):
        for s in (-1, 1):
            n = c.clone()
            n[:, ax] += s
            q = n // bsx
            k = slot[q[:, 0] + q[:, 1] * (nb + 2) + q[:, 2] * (nb + 2) ** 2]
            v = n % bsx
            near.append(torch.where(k >= 0, k * bsx ** 3 + v[:, 0] + v[:, 1] * bsx + v[:, 2] * bsx * bsx, cells).int())
    p = torch.zeros(cells + 1, device="cuda", dtype=torch.float64)
    b = b.double()
    x, r = torch.zeros_like(b), b.clone()
    p[:-1] = r
    rr = torch.dot(r, r)
    stop = 1e-24 * float(rr)
    for it in range(5000):
        ap = 6 * p[:-1]
        for n in near:
            ap -= p[n]
        alpha = rr / torch.dot(p[:-1], ap)
        x += alpha * p[:-1]
        r -= alpha * ap
        new = torch.dot(r, r)
        if it % 16 == 15 and float(new) <= stop:
            break
        p[:-1] = r + new / rr * p[:-1]
        rr = new
    return x


def _exact_poisson(case, seed):
    size, bsx = case["size"], case["bsx"]
    ids = _band_blocks(size // bsx, bsx, 0.35 * size, 16.0)
    return _solve64(ids, size // bsx, bsx, _smooth_rhs(seed, ids, size // bsx, bsx))


def _exact_batch(case, seed):
    groups = {}  # one per block size, in the order of the sizes' first problems
    for edge, bsx, ids, rhs in _batch_problems(case, seed):
        t = torch.from_numpy(ids.astype(np.int64)).cuda()
        groups.setdefault(bsx, []).append(_solve64(t, edge // bsx, bsx, rhs))
    return [torch.cat(x) for x in groups.values()]


def _exact_conv(case, seed):
    ids, nbr, x, dy, w, bias = _conv_inputs(case, seed)
    bs, cells = 1 << case["lg"], len(x)
    v = torch.arange(bs ** 3, device="cuda")
    c = torch.stack([v % bs, (v // bs) % bs, v // (bs * bs)], -1)
    xp = torch.cat([x.double(), torch.zeros((1, case["cin"]), device="cuda", dtype=torch.float64)])
    dp = torch.cat([dy.double(), torch.zeros((1, case["cout"]), device="cuda", dtype=torch.float64)])
    y = bias.double().repeat(cells, 1)
    dx = torch.zeros((cells, case["cin"]), device="cuda", dtype=torch.float64)
    dw = torch.empty((27, case["cout"], case["cin"]), device="cuda", dtype=torch.float64)
    for t in range(27):
        d = torch.tensor([t % 3 - 1, (t // 3) % 3 - 1, t // 9 - 1], device="cuda")
        src = {}
        for s in (1, -1):
            n = c + s * d
            o = n.div(bs, rounding_mode="floor") + 1
            k = nbr[:, o[:, 0] + 3 * o[:, 1] + 9 * o[:, 2]].long()
            m = n % bs
            src[s] = torch.where(k >= 0, k * bs ** 3 + m[:, 0] + m[:, 1] * bs + m[:, 2] * bs * bs, cells).reshape(-1)
        y += xp[src[1]] @ w[t].double().T
        dx += dp[src[-1]] @ w[t].double()
        dw[t] = dp[:-1].T @ xp[src[1]]
    return {"y": y.clamp(min=0), "dx": dx, "dw": dw}
