"""Density errors of a batch's scenes where a sum leaves the range of floats."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import PBFBatch, abi, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT


def _scene(n, mass=None):
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = 0.3 * H + 0.5 * H * g
    p = scenes.pbf_params(H, [0.0] * 3, [0.5 * m * H + H] * 3, n)
    if mass is not None:
        p.mass, p.rest_dens = mass, 1e-7  # 1e26: C is near 1e38
    return p, x


def test_scene_errors_past_the_range_of_floats(gpu):
    """Finite densities whose sum over a tile is no float, infinite ones, and an
    ordinary scene beside them: the means of C over the densities themselves, as
    doubles give them (1e-6: the roundings to a float of C and of the mean)."""
    scs = [_scene(700), _scene(600, 1e26), _scene(65, 1e26), _scene(300, 3e38), _scene(31)]
    b = PBFBatch([p for p, _ in scs], [len(x) for _, x in scs], iterations=1)
    b.set_particles(np.concatenate([x for _, x in scs]))
    b.step(0.0016)
    rho = b.get(abi.RX_DENSITY)
    for k, (p, x) in enumerate(scs):
        inv = np.float32(1) / np.float32(p.rest_dens)
        C = (b.scene(rho, k).astype(np.float64) * inv - 1).astype(np.float32)  # one rounding: a fused product
        want = [np.maximum(C, 0).astype(np.float64).mean(), np.abs(C).astype(np.float64).mean(), np.abs(C).max()]
        st = b.scene_stats(k)
        got = [st.density_error_one_sided, st.density_error_two_sided, st.density_error_max]
        assert np.isfinite(want).all() == (k != 3)
        np.testing.assert_allclose(got, want, rtol=1e-6)
    b.close()
