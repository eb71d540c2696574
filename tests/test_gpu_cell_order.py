"""The slot order of a grid build at the sizes where ranking inside the cells
can go wrong: one particle, cells of one, two and many particles, particles
that coincide, and everything clumped into a few cells.  The counting sort
ranks each cell's particles on the way through the gather; the radix sort
orders the 64-bit keys (cell << 32 | previous slot) themselves.  Both are the
same order, so a step from the same state is the same bit for bit."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxPBDSPH, rxSPH, scenes

pytestmark = pytest.mark.gpu


def _points(kind, n, box, rng):
    lo, hi = 0.05, box - 0.05
    x = np.zeros((n, 4), np.float32)
    if kind == "spread":
        x[:, :3] = rng.uniform(lo, hi, (n, 3))
    elif kind == "clumped":  # a few cells hold everything
        c = rng.uniform(0.2, box - 0.2, (3, 3))
        x[:, :3] = c[rng.integers(0, 3, n)] + rng.uniform(-0.02, 0.02, (n, 3))
    else:  # coincident pairs
        x[:, :3] = np.repeat(rng.uniform(lo, hi, ((n + 1) // 2, 3)), 2, axis=0)[:n]
    return x


@pytest.mark.parametrize("kind", ["spread", "clumped", "pairs"])
@pytest.mark.parametrize("n", [1, 2, 33, 257, 1500])
def test_ranked_and_radix_orders_step_identically(gpu, kind, n):
    rng = np.random.default_rng(n)
    p = scenes.wcsph_dam_break(8).params
    p.max_particles = n
    box = float(p.box_max[1])
    pos = _points(kind, n, box, rng)
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(0, 0.5, (n, 3))
    out = []
    for sort in (0, 1):
        q = abi.FsphParams.from_buffer_copy(p)
        q.grid_sort = sort
        ps = rxSPH(q)
        ps.Set(pos, vel)
        ps.Update(1e-4)
        ps.Update(1e-4)
        out.append([ps.GetArrayVBO(abi.RX_POSITION), ps.GetArrayVBO(abi.RX_VELOCITY),
                    ps.GetArrayVBO(abi.FSPH_SORTED_ID)])
        ps.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("side", [3, 16, 17, 203, 204])
def test_cell_table_scan_at_tile_edges(gpu, side):
    """The scan over the cell table takes one phase up to 4,096 cells, two up
    to 2,048 tiles of those and three past that: the neighbour sets of a few
    particles spread over the whole grid against brute force (whole numbers)."""
    h = 1.0
    p = scenes.pbf_params(h, [0.0] * 3, [1.0] * 3, 600)
    p.cell_skin = 0.0  # a cell is h (1 + 1e-3) wide, plus one cell of padding on each side
    for a in range(3):
        p.box_max[a] = (side - 2) * 1.001 * h * 0.9999
    p.particle_radius = 0.25
    rng = np.random.default_rng(side)
    n, top = 600, float(p.box_max[0])
    pos = np.zeros((n, 4), np.float32)
    c = rng.uniform(0, top, (60, 3))
    pos[:, :3] = np.clip(c[rng.integers(0, 60, n)] + rng.uniform(-1, 1, (n, 3)), 0, top)
    ps = rxPBDSPH(p)
    ps.Set(pos)
    off, idx = ps.GetNeights()
    ps.close()
    x = pos[:, :3].astype(np.float64)
    d2 = ((x[:, None] - x[None]) ** 2)
    near = (d2[..., 0] + d2[..., 1] + d2[..., 2]).astype(np.float32) <= np.float32(h * h)
    assert np.array_equal(np.diff(off), near.sum(1))
    assert np.array_equal(idx, np.nonzero(near)[1])
