"""Compressed fluid, whose candidates go through a tile of 1,024 in parts (four
warps for 32 slots) or past it: lists up to their limit and beyond, one cell of
everything, a particle far outside the box among the rest."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxPBDSPH, rxSPH, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT
U = 2.0 ** -24


def _positions(kind, n):
    rng = np.random.default_rng(n)
    x = np.zeros((n, 4), np.float32)
    if kind == "heap":  # all within a cell
        x[:, :3] = 1.0 + rng.uniform(0, 0.9 * H, (n, 3))
        return x
    s = 0.5 * H * float(kind)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x[:, :3] = 1.0 + s * (g + rng.uniform(-0.2, 0.2, (n, 3)))
    x[n // 2, :3] = 40.0  # where no tile reaches
    return x


@pytest.mark.parametrize("kind", ["0.85", "0.7", "0.55"])
@pytest.mark.parametrize("n", [5000, 20000, 33000])
def test_lists_step_as_the_cell_walk(gpu, kind, n):
    p = scenes.pbf_params(H, [0.9] * 3, [2.5] * 3, n, cell_skin=0.05)
    p.eta, p.min_iter, p.max_iter = 0.0, 2, 2
    x = _positions(kind, n)
    got = []
    for walk in (0, 1):
        q = abi.FsphParams.from_buffer_copy(p)
        q.walk_cells = walk
        ps = rxPBDSPH(q)
        ps.Set(x)
        ps.Update(0.0005)
        got.append([ps.GetArrayVBO(t) for t in (abi.RX_POSITION, abi.RX_VELOCITY, abi.RX_DENSITY)])
        ps.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind", ["0.85", "0.7", "0.55", "heap"])
@pytest.mark.parametrize("n", [1000, 12288, 13001, 30000, 66000])
def test_density_and_forces(gpu, kind, n):
    """Densities with lists and without are the same bits, and right: a term is
    rounded fewer than 20 times at its full size, a sum of k terms k times.  The
    forces from the lists and from the walks agree to the roundings of their terms:
    the sums of the two orders differ by k roundings of the terms' magnitudes."""
    if kind == "heap":
        n = min(n, 13001)
    x = _positions(kind, n)
    p = scenes.wcsph_dam_break(8).params
    p.max_particles = n
    for a in range(3):
        p.box_min[a], p.box_max[a] = 0.9, 2.5
    rng = np.random.default_rng(3)
    v = np.zeros_like(x)
    v[:, :3] = rng.normal(0, 1, (n, 3))
    got = []
    for walk in (0, 1):
        q = abi.FsphParams.from_buffer_copy(p)
        q.walk_cells = walk
        ps = rxSPH(q)
        got.append(ps.EvalForces(x, v))
        ps.close()
    (d, pr, a), (dw, _, aw) = got
    assert np.array_equal(d, dw)
    h, m, mu = float(np.float32(p.h)), float(p.mass), float(p.viscosity)
    x64, v64, d64, p64 = (t.astype(np.float64) for t in (x[:, :3], v[:, :3], d, pr))
    w = 315 / (64 * np.pi * h ** 9) * m
    for i in np.concatenate([[n // 2], rng.choice(n, 100, replace=False)]):
        dv = x64[i] - x64
        r = np.sqrt((dv ** 2).sum(1))
        near = r < h
        rho = w * ((h * h - r[near] ** 2) ** 3).sum()
        k = near.sum()
        assert abs(d64[i] - rho) <= U * k * (20 * w * h ** 6 + rho)
        j = near & (r > 0)
        gv = 45 / (np.pi * h ** 6)
        hr = h - r[j]
        ps2 = m * (abs(p64[i]) / d64[i] ** 2 + np.abs(p64[j]) / d64[j] ** 2)
        dvel = mu * m / d64[j] * np.abs(v64[j] - v64[i]).sum(1)
        big = (ps2 * gv * hr ** 2 + dvel * gv * hr).sum() + 10.0
        edge = (ps2 * gv * 2 * hr * h + dvel * gv * h).sum()
        assert np.abs(a[i, :3] - aw[i, :3]).max() <= 2 * U * ((k + 40) * big + 8 * edge)
