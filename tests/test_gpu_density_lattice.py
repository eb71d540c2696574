"""The density field on lattices whose bricks of nodes are cut off in every
way (one node, lines, sheets, ragged boxes), at kernel radii far from one, on
dense clumps whose candidates are evaluated in several goes, against 64-bit
sums.  The bar: up to 60 terms of one sign, each with a rounded distance
(1.5 x 2^-24 of r, at most 8e-8 of the term at r = 0) and a rounding of the
float sum (6e-8): 60 x 1.4e-7 = 8.4e-6 of the field's largest value."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import rxPBDSPH, scenes

pytestmark = pytest.mark.gpu


def _field(x, n, o, d, h, mass, lo, hi):
    ax = [o[a] + np.arange(n[a]) * d[a] for a in range(3)]
    z, y, xx = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    g = np.stack([xx, y, z], -1).reshape(-1, 3)
    out = np.zeros(len(g))
    aw = 315.0 / (64.0 * np.pi * h ** 9)
    for s in range(0, len(g), 512):
        r2 = ((g[s:s + 512, None] - x[None]) ** 2).sum(-1)
        out[s:s + 512] = mass * aw * (np.clip(h * h - r2, 0, None) ** 3).sum(1)
    return (out * np.all((g >= lo) & (g <= hi), axis=1)).reshape(n[2], n[1], n[0])


@pytest.mark.parametrize("h", [0.0457, 7e-4, 31.0])
@pytest.mark.parametrize("n", [(1, 1, 1), (37, 1, 1), (1, 1, 34), (3, 1, 9), (1, 21, 2), (19, 7, 5), (16, 12, 8)])
def test_lattices_against_64_bits(gpu, n, h):
    rng = np.random.default_rng(n[0] + 100 * n[1])
    m = 11
    s = 0.5 * h
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = np.zeros((m ** 3, 4), np.float32)
    x[:, :3] = (g + 0.8) * s + rng.uniform(-0.2, 0.2, (m ** 3, 3)) * s
    x[:60, :3] = x[60, :3] + rng.uniform(-0.2, 0.2, (60, 3)) * s  # a clump: more candidates than are kept
    box = [(m + 2) * s] * 3
    p = scenes.pbf_params(h, [0.0] * 3, box, m ** 3, particle_radius=0.25 * h)
    p.mass = scenes.lattice_mass(h, s)
    ps = rxPBDSPH(p)
    ps.Set(x)
    d = [1.02 * b / max(k - 1, 2) for b, k in zip(box, n)]
    o = [-0.008 * b if k > 2 else 0.4 * b for b, k in zip(box, n)]
    got = ps.CalImplicitField(n, o, d)
    ps.close()
    lo, hi = [-0.005 * b for b in box], [b + 0.005 * b for b in box]
    want = _field(x[:, :3].astype(np.float64), n, o, d, float(p.h), float(p.mass), lo, hi)
    top = _field(x[:, :3].astype(np.float64), (1, 1, 1), x[60, :3].astype(float), d, float(p.h), float(p.mass), lo,
                 hi).max()
    assert np.abs(got - want).max() <= 8.4e-6 * max(want.max(), 0.1 * top)


@pytest.mark.parametrize("d", [0.11, 0.5, 1.0, 1.3, 1.4, 2.2])
def test_spacings_on_both_sides_of_the_shared_bricks(gpu, d):
    """Nodes from far denser than the particles to ones that share no neighbour:
    the bricks' common set (in several goes where they are large) and the lanes'
    own walks."""
    h = 0.0457
    rng = np.random.default_rng(int(100 * d))
    m = 14
    s = 0.5 * h
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = np.zeros((m ** 3, 4), np.float32)
    x[:, :3] = (g + 0.8) * s + rng.uniform(-0.3, 0.3, (m ** 3, 3)) * s
    box = [(m + 2) * s] * 3
    p = scenes.pbf_params(h, [0.0] * 3, box, m ** 3, particle_radius=0.25 * h)
    p.mass = scenes.lattice_mass(h, s)
    ps = rxPBDSPH(p)
    ps.Set(x)
    n = [min(int(b / (d * h)), 22) for b in box]
    got = ps.CalImplicitField(n, [0.1 * h] * 3, [d * h] * 3)
    ps.close()
    lo, hi = [-0.005 * b for b in box], [b + 0.005 * b for b in box]
    want = _field(x[:, :3].astype(np.float64), n, [0.1 * h] * 3, [d * h] * 3, float(p.h), float(p.mass), lo, hi)
    assert np.abs(got - want).max() <= 8.4e-6 * want.max()
