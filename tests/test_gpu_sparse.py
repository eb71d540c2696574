"""Fluid on both sides of the density at which the lanes of a warp stop searching
their candidates together: spray, and a pool with spray above it (warps of either
kind, and warps half one and half the other), with one warp for 32 slots and with
four."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxPBDSPH, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT


def _scene(spacing, n, pool):
    """n particles at random, one in (spacing H)^3; with a pool, half of them a
    lattice at rest below the others."""
    rng = np.random.default_rng(n)
    k = n - n // 2 if pool else n
    side = spacing * H * k ** (1 / 3)
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = 0.3 * H + rng.uniform(0, side, (n, 3))
    if pool:
        m = max(1, int(side / (0.5 * H)))
        i = np.arange(n - k)
        x[k:, :3] = 0.3 * H + 0.5 * H * np.stack([i % m, i // (m * m), (i // m) % m], 1)
        x[:k, 1] += x[k:, 1].max()
    x = x[rng.permutation(n)]
    p = scenes.pbf_params(H, [0.0] * 3, (x[:, :3].max(0) + 0.3 * H).tolist(), n, cell_skin=0.1)
    p.eta, p.min_iter, p.max_iter = 0.0, 2, 3
    return p, x


@pytest.mark.parametrize("pool", [False, True])
@pytest.mark.parametrize("spacing", [0.8, 0.9, 1.0, 1.2, 2.0])
@pytest.mark.parametrize("n", [3000, 33000])
def test_lists_step_as_the_cell_walk(gpu, spacing, n, pool):
    """The same bits: what either meets beyond the other adds exact zeros."""
    p, x = _scene(spacing, n, pool)
    got = []
    for walk in (0, 1):
        q = abi.FsphParams.from_buffer_copy(p)
        q.walk_cells = walk
        ps = rxPBDSPH(q)
        ps.Set(x)
        for _ in range(2):
            ps.Update(0.0016)
        got.append([ps.GetArrayVBO(t) for t in (abi.RX_POSITION, abi.RX_VELOCITY, abi.RX_DENSITY)])
        ps.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("pool", [False, True])
@pytest.mark.parametrize("spacing", [0.8, 1.0, 2.0])
def test_neighbour_rows_against_brute_force(gpu, spacing, pool):
    p, x = _scene(spacing, 5001, pool)
    ps = rxPBDSPH(p)
    ps.Set(x)
    off, idx, d2 = ps.SetParticlesToCell(None, -1.0)
    ps.close()
    q = x[:, :3].astype(np.float64)
    h2 = np.float32(np.float32(p.h) * np.float32(p.h))
    for i0 in range(0, len(q), 1000):
        e = (q[i0:i0 + 1000, None] - q[None]) ** 2
        want = (e[..., 0] + e[..., 1] + e[..., 2]).astype(np.float32)
        near = want <= h2
        s = slice(off[i0], off[min(i0 + 1000, len(q))])
        assert np.array_equal(np.diff(off[i0:i0 + 1001]), near.sum(1))
        assert np.array_equal(idx[s], np.nonzero(near)[1])
        assert np.array_equal(d2[s], want[near])
