"""The one-kernel constraint loop (a graph step without a boundary) against the
host-driven loop of separate passes (use_graph = 0): the same positions,
velocities, densities, iteration counts, errors and grid builds bit for bit, at
block edges and on both sides of every size at which the launch shape changes."""
import threading

import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxPBDSPH, scenes

pytestmark = pytest.mark.gpu

H = scenes.H_DEFAULT


def _state(n, seed, squeeze=1.0, jitter=0.03):
    rng = np.random.default_rng(seed)
    m = max(2, int(np.ceil(n ** (1 / 3))))
    s = 0.5 * H * squeeze
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = np.zeros((n, 4), np.float32)
    x[:, :3] = 0.3 * H + g * s + rng.uniform(0, jitter * H, (n, 3))
    v = np.zeros_like(x)
    v[:, :3] = rng.normal(0, 0.5, (n, 3))
    p = scenes.pbf_params(H, [0.0] * 3, [1.5 * m * s + H] * 3, n)
    return p, x, v


def _run(p, x, v, steps, graph, boundary=None):
    q = abi.FsphParams.from_buffer_copy(p)
    q.use_graph = graph
    ps = rxPBDSPH(q)
    ps.Set(x, v)
    if boundary is not None:
        ps.SetBoundary(boundary)
    rec = []
    for _ in range(steps):
        ps.Update(0.0016)
        st = ps.last_stats
        rec.append((st.iterations, st.grid_builds, st.density_error_one_sided, st.density_error_two_sided,
                    st.density_error_max, st.status))
    out = [ps.GetArrayVBO(t) for t in (abi.RX_POSITION, abi.RX_VELOCITY, abi.RX_DENSITY, abi.RX_SCALING_FACTOR,
                                       abi.RX_PREDICT_POS)]
    ps.close()
    return rec, out


def _same(p, x, v, steps=2):
    a, b = _run(p, x, v, steps, 1), _run(p, x, v, steps, 0)
    assert a[0] == b[0]
    assert all(np.array_equal(s, t) for s, t in zip(a[1], b[1]))
    return a[0]


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 1000, 6912, 19456, 19457, 38912, 38913, 65535, 65536,
                               65537])
def test_fixed_iterations(gpu, n):
    p, x, v = _state(n, n)
    p.eta, p.min_iter, p.max_iter, p.error_mode = 0.0, 2, 5, abi.ERR_TWO_SIDED  # |C| > 0: never below eta
    assert [r[0] for r in _same(p, x, v)] == [5, 5]


@pytest.mark.parametrize("mode", [abi.ERR_ONE_SIDED, abi.ERR_TWO_SIDED])
@pytest.mark.parametrize("clamp", [0, 1])
@pytest.mark.parametrize("min_iter", [0, 1, 4])
def test_tolerance_decides(gpu, mode, clamp, min_iter):
    p, x, v = _state(3000, 5)
    p.error_mode, p.clamp_constraint, p.min_iter, p.max_iter = mode, clamp, min_iter, 60
    p.eta = 2e-3 if mode == abi.ERR_ONE_SIDED else 5e-2
    rec = _same(p, x, v, 3)
    assert all(r[0] >= max(min_iter, 1) for r in rec)


@pytest.mark.parametrize("kahan", [0, 1])
@pytest.mark.parametrize("ext", [0, 1])
def test_rebuilds_inside_the_loop_and_overflowed_lists(gpu, kahan, ext):
    """A squeezed block flies apart (grid rebuilds between two launches of the
    loop, and after it), its lists overflow (cell walks)."""
    p, x, v = _state(4000, 9, squeeze=0.72)
    p.eta, p.min_iter, p.max_iter, p.cell_skin, p.compensated_density = 0.0, 2, 12, 0.03, kahan
    if not ext:
        p.xsph_c = p.vort_eps = 0.0
    rec = _same(p, x, v, 4)
    assert max(r[1] for r in rec) > 2


def test_many_iterations_and_the_cap(gpu):
    p, x, v = _state(2000, 3, squeeze=0.9)
    p.eta, p.min_iter, p.max_iter, p.clamp_constraint = 1e-9, 2, 150, 1
    rec = _same(p, x, v, 1)
    assert rec[0][0] == 150 and rec[0][5] == abi.NOT_CONVERGED


def test_contexts_step_side_by_side(gpu):
    """Two contexts from two host threads, each its own stream and counters."""
    p, x, v = _state(9000, 11)
    p.eta, p.min_iter, p.max_iter = 0.0, 2, 8
    want = _run(p, x, v, 20, 0)
    got = [None, None]

    def go(k):
        got[k] = _run(p, x, v, 20, 1)

    ts = [threading.Thread(target=go, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for g in got:
        assert g[0] == want[0] and all(np.array_equal(a, b) for a, b in zip(g[1], want[1]))


@pytest.mark.parametrize("n", [69632, 155649, 233473, 300007, 500001])
def test_swept_scenes(gpu, n):
    """More particles than the loop keeps on threads of their own: less than one
    round of the resident warps, one and a little, more, a ragged last chunk."""
    p, x, v = _state(n, n)
    p.eta, p.min_iter, p.max_iter, p.error_mode = 0.0, 2, 4, abi.ERR_TWO_SIDED
    assert [r[0] for r in _same(p, x, v)] == [4, 4]


@pytest.mark.parametrize("kahan", [0, 1])
def test_swept_scene_with_rebuilds_and_overflowed_lists(gpu, kahan):
    p, x, v = _state(80000, 9, squeeze=0.72)
    p.eta, p.min_iter, p.max_iter, p.cell_skin, p.compensated_density = 0.0, 2, 12, 0.03, kahan
    rec = _same(p, x, v, 3)
    assert max(r[1] for r in rec) > 2


@pytest.mark.parametrize("mode", [abi.ERR_ONE_SIDED, abi.ERR_TWO_SIDED])
def test_swept_scene_stops_at_its_tolerance(gpu, mode):
    p, x, v = _state(90000, 5)
    p.error_mode, p.min_iter, p.max_iter, p.eta = mode, 2, 60, 5e-3 if mode == abi.ERR_ONE_SIDED else 5e-2
    _same(p, x, v, 2)


def test_boundary_passes_on_both_sides_of_their_change_of_form(gpu):
    """57,344 particles beside a shell, and the same with one more far away, which
    takes the other form of the constraint passes: the same bits for all the rest."""
    n = 57344
    p, x, v = _state(n, 4)
    far = np.zeros((1, 4), np.float32)
    far[0, :3] = np.array(list(p.box_max)[:3]) - H
    p.eta, p.min_iter, p.max_iter = 0.0, 2, 3
    mid = 0.5 * (x[:, :3].min(0) + x[:, :3].max(0)) - 0.05
    b = scenes.box_surface([float(c) for c in mid], 0.1, 0.3 * H)
    got = []
    for y, w in ((x, v), (np.concatenate([x, far]), np.concatenate([v, 0 * far]))):
        q = abi.FsphParams.from_buffer_copy(p)
        q.max_particles = len(y)
        got.append(_run(q, y, w, 2, 1, b)[1])
    for s, t in zip(*got):
        assert np.array_equal(s[:n], t[:n])
