"""The slot order of a grid build at the sizes where ranking inside the cells
can go wrong: one particle, cells of one, two and many particles, particles
that coincide, and everything clumped into a few cells.  The counting sort
ranks each cell's particles on the way through the gather; the radix sort
orders the 64-bit keys (cell << 32 | previous slot) themselves.  Both are the
same order, so a step from the same state is the same bit for bit."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxSPH, scenes

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
