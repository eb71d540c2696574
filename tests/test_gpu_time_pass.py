"""fsph_time_pass of the loop kernel: a time on every form, refused beside a
boundary and without lists, and the steps after it as without it."""
import ctypes

import numpy as np
import pytest

from fltk_sph_ice_gb300 import abi, rxPBDSPH, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [(6, 6, 12), (16, 16, 32), (32, 32, 64)])
def test_loop_pass(gpu, block):
    sc = scenes.pbf_double_dam_break(block=block)
    out = []
    for timed in (False, True):
        ps = rxPBDSPH(sc.params)
        ps.Set(sc.pos, sc.vel)
        t = ctypes.c_float(0)
        if timed:
            assert ps.L.fsph_time_pass(ps._ctx, abi.PASS_LOOP, 7, ctypes.byref(t)) == abi.OK
            assert 0 < t.value < 100
            ps.Set(sc.pos, sc.vel)
        ps.Update(sc.dt)
        out.append((ps.last_stats.iterations, ps.GetArrayVBO(abi.RX_POSITION)))
        ps.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])


def test_loop_pass_is_refused_where_no_step_runs_it(gpu):
    sc = scenes.pbf_double_dam_break(block=(6, 6, 12))
    t = ctypes.c_float(0)
    ps = rxPBDSPH(sc.params)
    ps.Set(sc.pos, sc.vel)
    ps.SetBoundary(scenes.box_surface([0.3, 0.1, 0.3], 0.05, 0.3 * scenes.H_DEFAULT))
    assert ps.L.fsph_time_pass(ps._ctx, abi.PASS_LOOP, 3, ctypes.byref(t)) == abi.UNSUPPORTED
    ps.close()
    p = abi.FsphParams.from_buffer_copy(sc.params)
    p.walk_cells = 1
    ps = rxPBDSPH(p)
    ps.Set(sc.pos, sc.vel)
    assert ps.L.fsph_time_pass(ps._ctx, abi.PASS_LOOP, 3, ctypes.byref(t)) == abi.UNSUPPORTED
    ps.close()
