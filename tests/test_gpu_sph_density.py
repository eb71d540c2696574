"""The WCSPH density pass on both sides of the sizes where it changes form, with
full and ragged warps, sparse fluid (a warp's slots in many cells) and clumps
(more neighbours than a list or a tile holds): density, and the forces of the
lists that the pass leaves, against 64 bits."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxSPH, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT
U = 2.0 ** -24


def _scene(kind, n):
    rng = np.random.default_rng(n)
    x = np.zeros((n, 4), np.float32)
    if kind == "lattice":
        m = int(np.ceil(n ** (1 / 3)))
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        x[:, :3] = 0.3 * H + 0.5 * H * (g + rng.uniform(-0.1, 0.1, (n, 3)))
    elif kind == "sparse":
        x[:, :3] = rng.uniform(0.3 * H, 3.0, (n, 3))
    else:  # 64 clumps of n / 64 slots, a third of them outside a clump
        c = rng.uniform(0.3, 2.7, (64, 3))
        x[:, :3] = c[rng.integers(0, 64, n)] + rng.normal(0, 0.6 * H, (n, 3))
        x[::3, :3] = rng.uniform(0.3, 2.7, (len(x[::3]), 3))
    p = scenes.wcsph_dam_break(8).params
    p.max_particles = n
    hi = x[:, :3].max(0) + 0.3 * H
    p.box_max = type(p.box_max)(*hi.tolist(), *([0.0] * (len(p.box_max) - 3)))
    v = np.zeros((n, 4), np.float32)
    v[:, :3] = rng.normal(0, 1, (n, 3))
    return p, x, v


@pytest.mark.parametrize("kind", ["lattice", "sparse", "clumped"])
@pytest.mark.parametrize("n", [1, 33, 5000, 9000, 12287, 12288, 32767, 32801, 65536, 65537])
def test_density_and_forces_against_64_bits(gpu, kind, n):
    """A density term (h^2 - r^2)^3 <= h^6 is rounded fewer than 20 times at its
    full size, a sum of k terms k times at most; a force term is rounded fewer
    than 40 times (rsqrtf is good to 2 ulp) and h - r carries the rounding of
    h beside; the forces start from the pass's own density and pressure."""
    p, x, v = _scene(kind, n)
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
    for i in np.random.default_rng(1).choice(n, min(n, 200), replace=False):
        dv = x64[i] - x64
        r = np.sqrt((dv ** 2).sum(1))
        near = r < h
        w = 315 / (64 * np.pi * h ** 9) * m
        rho = w * ((h * h - r[near] ** 2) ** 3).sum()
        k = near.sum()
        assert abs(d64[i] - rho) <= U * k * (20 * w * h ** 6 + rho)
        near &= r > 0
        dv, r, j = dv[near], r[near], near
        g = -45 / (np.pi * h ** 6) * (h - r) ** 2 / r
        fp = -m * ((p64[i] / d64[i] ** 2 + p64[j] / d64[j] ** 2) * g)[:, None] * dv
        fv = mu * m * ((45 / (np.pi * h ** 6) * (h - r)) / d64[j])[:, None] * (v64[j] - v64[i])
        gv = 45 / (np.pi * h ** 6)
        ps2 = m * (abs(p64[i]) / d64[i] ** 2 + np.abs(p64[j]) / d64[j] ** 2)
        dvel = mu * m / d64[j] * np.abs(v64[j] - v64[i]).sum(1)
        big = (ps2 * gv * (h - r) ** 2 + dvel * gv * (h - r)).sum() + 10.0
        edge = (ps2 * gv * 2 * (h - r) * h + dvel * gv * h).sum()
        want = fp.sum(0) + fv.sum(0) + np.array(list(p.gravity)[:3], np.float64)
        for f in (a, aw):
            assert np.abs(f[i, :3] - want).max() <= U * ((k + 40) * big + 8 * edge)
