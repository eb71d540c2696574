"""The neighbour lists of the warp-wide build where it can go wrong: warps that
are not full, warps whose slots lie in many rows of cells (sparse fluid, thin
tanks), clumps whose candidates overflow a list or a warp's tile.  A pass over
the lists and a walk over the 27 cells meet the same neighbours in the same
ascending order, and what else either meets adds exact zeros, so a step with
lists equals the same step walking the cells bit for bit."""
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
@pytest.mark.parametrize("n", [1, 31, 32, 33, 161, 2500])
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
