"""The neighbour lists of the warp-wide build where it can go wrong: warps that
are not full, warps whose slots lie in many rows of cells (sparse fluid, thin
tanks), clumps whose candidates overflow a list or a warp's tile.  A pass over
the lists and a walk over the 27 cells meet the same neighbours in the same
ascending order, and what else either meets adds exact zeros, so a step with
lists equals the same step walking the cells bit for bit."""
import ctypes

import numpy as np
import pytest

from fltk_sph_ice_gb300 import PBFBatch, abi, rxPBDSPH, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT


def _scene(kind, n, seed):
    rng = np.random.default_rng(seed)
    box = {"thin": [1.5, 0.05, 0.05], "flat": [0.6, 0.06, 0.6]}.get(kind, [0.7, 0.6, 0.5])
    lo, hi = np.full(3, 0.3 * H), np.array(box) - 0.3 * H
    x = np.zeros((n, 4), np.float32)
    if kind == "clumped":
        c = rng.uniform(lo, hi, (4, 3))
        x[:, :3] = np.clip(c[rng.integers(0, 4, n)] + rng.normal(0, 0.3 * H, (n, 3)), lo, hi)
    elif kind == "dense":  # a lattice four times as dense as at rest, ragged at the end
        s = 0.5 * H / 4 ** (1 / 3)
        m = int(np.ceil(n ** (1 / 3)))
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        x[:, :3] = np.clip(lo + g * s + rng.uniform(-0.1, 0.1, (n, 3)) * s, lo, hi)
    else:
        x[:, :3] = rng.uniform(lo, hi, (n, 3))
    p = scenes.pbf_params(H, [0.0] * 3, box, n, cell_skin=0.1)
    p.eta, p.min_iter, p.max_iter = 0.0, 2, 3
    return p, x


@pytest.mark.parametrize("kind", ["sparse", "thin", "flat", "clumped", "dense"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 161, 2500, 32768, 32801])
def test_lists_step_as_the_cell_walk(gpu, kind, n):
    p, x = _scene(kind, n, n)
    got = []
    for walk in (0, 1):
        q = abi.FsphParams.from_buffer_copy(p)
        q.walk_cells = walk
        ps = rxPBDSPH(q)
        ps.Set(x)
        try:
            ps.Update(0.0016)
            ps.Update(0.0016)
        except abi.FsphError as e:  # a clump may diverge; both then do
            got.append(e.status)
        else:
            got.append(np.concatenate([ps.GetArrayVBO(t) for t in (abi.RX_POSITION, abi.RX_VELOCITY)]))
        ps.close()
    assert np.array_equal(np.asarray(got[0]), np.asarray(got[1]))


def test_batched_lists_do_not_depend_on_the_tiles(gpu):
    """Tiles of every size, ragged ends, a scene of one particle: the lists,
    and so the step, are the same."""
    scs = [_scene("sparse", n, n) for n in (1, 130, 700)] + [_scene("dense", 515, 3)]
    got = []
    for block in (128, 256, 512):
        b = PBFBatch([p for p, _ in scs], [x.shape[0] for _, x in scs], iterations=3)
        b.set_config(block, 1, 0.1)
        b.set_particles(np.concatenate([x for _, x in scs]))
        b.step(0.0016)
        got.append(b.get(abi.RX_POSITION))
        b.close()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


@pytest.mark.parametrize("kind", ["sparse", "thin", "clumped", "dense"])
@pytest.mark.parametrize("n", [1, 33, 900])
def test_neighbour_rows_against_brute_force(gpu, kind, n):
    """Rows of no, one, up to 64 (one or two a lane) and more neighbours (the
    clumps), of the context's particles and of given positions, whole numbers
    and squared distances equal to the reference criterion's."""
    p, x = _scene(kind, n, 7 * n)
    ps = rxPBDSPH(p)
    ps.Set(x)
    ps.Update(0.0016) if kind == "sparse" else None  # a slot order that is not the particles'
    for prts, h in ((None, -1.0), (x[::-1].copy(), 0.8 * H)):
        off, idx, d2 = ps.SetParticlesToCell(prts, h)
        q = (ps.GetArrayVBO(abi.RX_POSITION) if prts is None else prts)[:, :3].astype(np.float64)
        r = np.float32(p.h if h < 0 else h)
        e = (q[:, None] - q[None]) ** 2
        want = (e[..., 0] + e[..., 1] + e[..., 2]).astype(np.float32)
        near = want <= np.float32(r * r)
        assert np.array_equal(np.diff(off), near.sum(1))
        assert np.array_equal(idx, np.nonzero(near)[1])
        assert np.array_equal(d2, want[near])
    ps.close()


@pytest.mark.parametrize("n", [1, 31, 700, 1024, 1025, 8192, 8193, 20000, 40000, 65536])
def test_allocation_free_lambda_at_every_lane_count(gpu, n):
    """The allocation-free pass takes 32 to 4 lanes a particle by size; density
    and lambda against 64 bits.  The bars: a sum of about 30 terms of one sign,
    each rounded a few times (1e-6 of the density); lambda has that error
    divided by |C| >= 0.1 here and the error of its denominator (2e-5)."""
    import torch
    rng = np.random.default_rng(n)
    s = 0.5 * H * 0.9  # compressed: C is far from zero
    m = int(np.ceil(n ** (1 / 3)))
    x = np.zeros((n, 4), np.float32)
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x[:, :3] = 0.3 * H + g * s + rng.uniform(-0.05, 0.05, (n, 3)) * s
    p = scenes.pbf_params(H, [0.0] * 3, [m * s + 0.6 * H] * 3, n)
    t = torch.from_numpy(x).cuda()
    d, lam = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    ptr = lambda a: ctypes.c_void_p(a.data_ptr())  # noqa: E731
    L = abi.lib()
    L.fsph_pbf_eval_lambda_noalloc.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_int] + [ctypes.c_void_p] * 3
    torch.cuda.synchronize()
    assert L.fsph_pbf_eval_lambda_noalloc(ctypes.byref(p), ptr(t), n, ptr(d), ptr(lam), None) == abi.OK
    torch.cuda.synchronize()
    at = rng.choice(n, min(n, 300), replace=False)  # rows checked against every particle
    h = float(np.float32(p.h))
    q = t[:, :3].double()
    dv = q[torch.from_numpy(at).cuda()][:, None] - q[None]
    r = dv.square().sum(-1).sqrt()
    rho = float(p.mass) * 315 / (64 * np.pi * h ** 9) * (h * h - r * r).clamp(min=0).pow(3).sum(1)
    gr = torch.where(r > 0, 45 / (np.pi * h ** 6) * (h - r).clamp(min=0).square() / r.clamp(min=1e-12),
                     torch.zeros_like(r)) / p.rest_dens
    gd = gr[..., None] * dv
    sd = gd.square().sum((1, 2)) + gd.sum(1).square().sum(1)
    want = -(rho / p.rest_dens - 1) / (sd + p.epsilon)
    at = torch.from_numpy(at).cuda()
    assert ((d[at] - rho).abs() <= 1e-6 * rho).all()
    keep = (rho / p.rest_dens - 1).abs() >= 0.1
    assert keep.any() or n < 700
    assert ((lam[at] - want).abs() <= 2e-5 * want.abs())[keep].all()
