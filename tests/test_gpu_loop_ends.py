"""How the one-kernel constraint loop ends when it does not end at its tolerance
(a density that is not a number, a barrier's wait that runs out), and that graph
steps without a boundary do run it."""
import numpy as np
import pytest

from fltk_sph_ice_gb300 import FsphError, abi, rxPBDSPH, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT
FORMS = [6912, 30000, 60000, 69632]  # blocks of 64, 128, 256; the sweep


def _scene(n, h=H, **kw):
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1 / 3)))
    s = 0.5 * h
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = 0.3 * h + g * s + rng.uniform(0, 0.02 * h, (n, 3))
    p = scenes.pbf_params(h, [0.0] * 3, [1.5 * m * s + h] * 3, n, **kw)
    p.cell_skin = 0.2
    return p, x


def _arrays(ps):
    return [ps.GetArrayVBO(t) for t in (abi.RX_POSITION, abi.RX_VELOCITY, abi.RX_DENSITY, abi.RX_SCALING_FACTOR)]


def _fixed(p, iterations, graph=1):
    q = abi.FsphParams.from_buffer_copy(p)
    q.eta, q.min_iter, q.max_iter, q.error_mode, q.use_graph = 0.0, 2, iterations, abi.ERR_TWO_SIDED, graph
    return q


@pytest.mark.parametrize("boundary", [False, True])
@pytest.mark.parametrize("n", FORMS)
def test_iterations_are_no_launches(gpu, n, boundary):
    """Steps of 3 and of 9 iterations on one grid build launch as many kernels; with
    a boundary (which the loop kernel does not take) 3 more an iteration."""
    p, x = _scene(n)
    got = []
    for it in (3, 9):
        ps = rxPBDSPH(_fixed(p, it))
        ps.Set(x)
        if boundary:
            ps.SetBoundary(scenes.box_surface([float(p.box_max[0]) - 0.1] * 3, 0.05, 0.3 * H))
        ps.Update(1e-4)
        st = ps.last_stats
        assert (st.iterations, st.grid_builds) == (it, 1)
        got.append(st.kernels)
        ps.close()
    assert got[1] - got[0] == (18 if boundary else 0)


@pytest.mark.parametrize("n", FORMS)
def test_a_density_that_is_not_a_number_stops_it(gpu, n):
    """h = 1e-8: the kernel's coefficient is infinite and the terms underflow to
    zero, so every density is not a number.  Both forms stop at the first
    iteration, report it and leave the same arrays."""
    p, x = _scene(n, 1e-8)
    got = []
    for graph in (1, 0):
        ps = rxPBDSPH(_fixed(p, 5, graph))
        ps.Set(x)
        with pytest.raises(FsphError) as e:
            ps.Update(1e-4)
        assert e.value.status == abi.NAN_DETECTED
        st = ps.last_stats
        got.append(([st.iterations, st.grid_builds, st.density_error_max, st.density_error_one_sided], _arrays(ps)))
        ps.close()
    assert got[0][0][0] == 1
    np.testing.assert_array_equal(got[0][0], got[1][0])
    for a, b in zip(got[0][1], got[1][1]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", FORMS)
def test_a_wait_that_runs_out(gpu, n):
    """Blocks that look once for the others give up: the step says so, and the next
    one, with the limit back, is as if nothing had been."""
    p, x = _scene(n)
    ref = rxPBDSPH(_fixed(p, 10))
    ref.Set(x)
    ref.Update(1e-4)
    ps = rxPBDSPH(_fixed(p, 10))
    assert ps.L.fsph_set_wait_limit(ps._ctx, -1) == abi.INVALID_ARG
    for _ in range(2):
        assert ps.L.fsph_set_wait_limit(ps._ctx, 1) == abi.OK
        ps.Set(x)
        with pytest.raises(FsphError) as e:
            ps.Update(1e-4)
        assert e.value.status == abi.TIMEOUT and "barrier" in str(e.value)
        assert ps.L.fsph_set_wait_limit(ps._ctx, 0) == abi.OK
        ps.Set(x)
        ps.Update(1e-4)
        assert ps.last_stats.iterations == 10
        for a, b in zip(_arrays(ps), _arrays(ref)):
            np.testing.assert_array_equal(a, b)
    ps.close()
    ref.close()
