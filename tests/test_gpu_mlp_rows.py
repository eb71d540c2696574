"""Every row of a batch reaches the training gradient: with targets that the
network already meets in all rows but one, the gradient is that row's, at the
edges of a warp's 16 rows, of a block's 64 and of the blocks' rounds."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 64, 65, 304 * 64, 304 * 64 + 1, 700 * 64 - 5])
def test_one_row_gradient(gpu, n):
    """The bar: an activation and a delta of a product may each round to BF16 the
    other way (2^-8), and the delta's own two products before it."""
    from fltk_sph_ice_gb300.warmstart import WarmStartNet, init_blob
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, omlp.NI)).astype(np.float32)
    blob = init_blob(rng.standard_normal((64, omlp.NI)).astype(np.float32),
                     (rng.standard_normal((64, 3)) * 0.02).astype(np.float32), seed=3)
    blob[omlp.O_B1:omlp.O_W2] = rng.standard_normal(64) * 0.1
    blob[omlp.O_B2:omlp.O_W3] = rng.standard_normal(64) * 0.1
    net = WarmStartNet(blob)
    y = np.asarray(net.forward(x), np.float32)
    for row in sorted({0, n // 2, n - 1, min(n - 1, 304 * 64 - 1)}):
        t = y.copy()
        t[row] += np.float32(0.05) * (1 + np.arange(3, dtype=np.float32))
        g, _ = net.gradient(x, t)
        want, _ = omlp.gradient(blob, x[row:row + 1], t[row:row + 1], bf16_emul=True)
        want = np.asarray(want, np.float64) / n
        for a, b in ((omlp.O_W1, omlp.O_B1), (omlp.O_B1, omlp.O_W2), (omlp.O_W2, omlp.O_B2), (omlp.O_B2, omlp.O_W3),
                     (omlp.O_W3, omlp.O_B3), (omlp.O_B3, omlp.O_SCALE)):
            assert np.abs(g[a:b] - want[a:b]).max() <= 4 * 2.0 ** -8 * np.abs(want[a:b]).max()
