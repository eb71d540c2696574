"""The density lattice of a collapsing dam against the oracle, which every host
has (the comparison with the reference's own code is in test_gpu_density_grid.py)."""
import numpy as np
import pytest

import oracle
from fltk_sph_ice_gb300 import abi, rxPBDSPH, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [(96, 30, 50), (33, 7, 9)])
def test_density_lattice_matches_the_oracle(gpu, nodes):
    """The bar of the comparison with the reference's code: 1e-6 of the largest value."""
    from test_density_grid_oracle import lattice
    sc = scenes.pbf_double_dam_break(block=(16, 16, 32))
    p = sc.params
    ps = rxPBDSPH(p)
    ps.Set(sc.pos, sc.vel)
    for _ in range(30):
        ps.Update(sc.dt)
    x = ps.GetArrayVBO(abi.RX_POSITION)
    nn, lo, d = lattice(p, nodes)
    got = ps.CalImplicitField(nn, lo, d)
    o = oracle.Oracle(p, sc.n, threads=4)
    o.set(x)
    want = o.density_grid(nn, lo, d)
    assert (want > 0).any()
    assert np.abs(got - want).max() <= 1e-6 * want.max()
    k, j, i = (np.array(got.shape) // 2).tolist()
    pt = [lo[0] + i * d[0], lo[1] + j * d[1], lo[2] + k * d[2]]
    assert abs(ps.GetImplicit(*pt) - got[k, j, i]) <= 1e-6 * want.max()
    ps.close()
