"""A heap in the last cell of the box with one particle far outside it, which the
grid keeps in that same cell: the last part of a turn finds a candidate that the
tile cannot hold, and what the earlier parts gave has to be forgotten."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxPBDSPH, rxSPH, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT
U = 2.0 ** -24


def _corner(n, hi=2.5):
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = hi - 0.3 * H - np.random.default_rng(n).uniform(0, 0.25 * H, (n, 3))
    x[-1, :3] = 40.0
    return x


@pytest.mark.parametrize("n", [3000, 13001, 66000])
def test_density(gpu, n):
    """The bar of the other density tests: a term is rounded fewer than 20 times
    at its full size, a sum of k terms k times."""
    x = _corner(n)
    p = scenes.wcsph_dam_break(8).params
    p.max_particles = n
    for a in range(3):
        p.box_min[a], p.box_max[a] = 2.0, 2.5
    got = []
    for walk in (0, 1):
        q = abi.FsphParams.from_buffer_copy(p)
        q.walk_cells = walk
        ps = rxSPH(q)
        got.append(ps.EvalForces(x, np.zeros_like(x))[0])
        ps.close()
    d = got[0]
    assert np.array_equal(d, got[1])
    h, x64 = float(np.float32(p.h)), x[:, :3].astype(np.float64)
    w = 315 / (64 * np.pi * h ** 9) * float(p.mass)
    for i in np.concatenate([[0, n - 2, n - 1], np.random.default_rng(1).choice(n, 30, replace=False)]):
        r2 = ((x64[i] - x64) ** 2).sum(1)
        k = (r2 < h * h).sum()
        rho = w * ((h * h - r2[r2 < h * h]) ** 3).sum()
        assert abs(d[i] - rho) <= U * k * (20 * w * h ** 6 + rho)


@pytest.mark.parametrize("n", [1500, 2500])
def test_neighbour_rows_and_lists(gpu, n):
    x = _corner(n)
    p = scenes.pbf_params(H, [2.0] * 3, [2.5] * 3, n, cell_skin=0.05)
    p.eta, p.min_iter, p.max_iter = 0.0, 2, 2
    ps = rxPBDSPH(p)
    ps.Set(x)
    off, idx, d2 = ps.SetParticlesToCell(None, -1.0)
    ps.close()
    q = x[:, :3].astype(np.float64)
    e = (q[:, None] - q[None]) ** 2
    want = (e[..., 0] + e[..., 1] + e[..., 2]).astype(np.float32)
    near = want <= np.float32(np.float32(p.h) * np.float32(p.h))
    assert np.array_equal(np.diff(off), near.sum(1))
    assert np.array_equal(idx, np.nonzero(near)[1]) and np.array_equal(d2, want[near])
