"""compensated_density in the allocation-free lambda pass: positions on a grid of
1/16 with h = 1 make every density term a multiple of 2^-24 that single precision
holds exactly, so a density is in error by its sum alone."""
import ctypes

import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


def _density(n, compensated):
    """the pass's density sums over mass aw, and the sums themselves (64 bits)"""
    import torch
    rng = np.random.default_rng(n)
    side = max(2, int(np.ceil((n / 60) ** (1 / 3))))  # 60 particles a unit of volume, some 250 within h
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = rng.integers(0, 16 * side, (n, 3)) / 16.0 + 1.0
    p = scenes.pbf_params(1.0, [0.0] * 3, [side + 2.0] * 3, n, mass=1.0, rest_dens=300.0)
    p.compensated_density = compensated
    t = torch.from_numpy(x).cuda()
    d, lam = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    L = abi.lib()
    L.fsph_pbf_eval_lambda_noalloc.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_int] + [ctypes.c_void_p] * 3
    torch.cuda.synchronize()
    assert L.fsph_pbf_eval_lambda_noalloc(ctypes.byref(p), t.data_ptr(), n, d.data_ptr(), lam.data_ptr(),
                                          None) == abi.OK
    torch.cuda.synchronize()
    at = torch.from_numpy(rng.choice(n, min(n, 2000), replace=False)).cuda()
    q = t[:, :3].double()
    want = torch.cat([(1.0 - (q[a][:, None] - q[None]).square().sum(-1)).clamp(min=0).pow(3).sum(1)
                      for a in at.split(200)])
    c = float(np.float32(315 / (64 * np.pi)))  # mass aw, one single-precision factor
    return d[at].double() / c, want


@pytest.mark.parametrize("n", [200, 1024, 7000, 8193, 20000, 40000, 65536])
def test_compensated_sums_at_every_lane_count(gpu, n):
    """32 to 4 lanes a particle.  The bar: the sum and its product with mass aw
    are each rounded once (2^-24 each; the compensation's own error, 2^-48 a
    term, is far below).  A plain sum of 250 terms is past it for some particle."""
    got, want = _density(n, 1)
    assert ((got - want).abs() <= 2.001 * 2.0 ** -24 * want).all()
    plain, _ = _density(n, 0)
    assert ((plain - want).abs() > 2.001 * 2.0 ** -24 * want).any() or n < 1000
