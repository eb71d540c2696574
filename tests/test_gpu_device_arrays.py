"""fsph_set_array / fsph_get_array on device memory: the kernels read and write
the caller's memory themselves where it is an aligned range of one allocation,
and go through a copy otherwise (a misaligned view, one of the context's own
arrays); the values are the same, and a range that holds a NaN is still
rejected with the state unchanged."""
import ctypes

import numpy as np
import pytest

from fltk_sph_ice_gb300 import PBFBatch, abi, rxPBDSPH, scenes

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("block", [(2, 2, 2), (5, 3, 7), (12, 12, 24)])
def test_device_arrays_equal_host_arrays(gpu, block, offset):
    import torch
    sc = scenes.pbf_double_dam_break(block=block)
    ps = rxPBDSPH(sc.params)
    ps.Set(sc.pos, sc.vel)
    ps.Update(sc.dt)
    n = sc.n
    rng = np.random.default_rng(n)
    buf = torch.full((4 * n + 8,), -7.0, device="cuda")
    view = buf[offset:offset + 4 * n]  # offset 1: four bytes past a 16-byte boundary
    start, count = n // 3, n - n // 3 - 1
    for which in (abi.RX_POSITION, abi.RX_VELOCITY):
        new = ps.GetArrayVBO(which)
        new[:, :3] += rng.uniform(-1e-3, 1e-3, (n, 3)).astype(np.float32)
        view.copy_(torch.from_numpy(new.reshape(-1)))
        torch.cuda.synchronize()
        st = ps.L.fsph_set_array(ps.handle, which, ctypes.c_void_p(view.data_ptr() + 16 * start), start, count,
                                 abi.DEVICE)
        assert st == abi.OK
        now = ps.GetArrayVBO(which)
        assert np.array_equal(now[start:start + count], new[start:start + count])
    for which, width in ((abi.RX_POSITION, 4), (abi.RX_VELOCITY, 4), (abi.RX_DENSITY, 1), (abi.RX_ATTRIBUTE, 1),
                         (abi.FSPH_SORTED_ID, 1), (abi.RX_SCALING_FACTOR, 1), (abi.RX_PREDICT_POS, 4)):
        buf.fill_(-7.0)
        torch.cuda.synchronize()
        assert ps.L.fsph_get_array(ps.handle, which, _p(view), abi.DEVICE, None) == abi.OK
        want = ps.GetArrayVBO(which)
        got = view[:width * n].cpu().numpy().view(want.dtype).reshape(want.shape)
        assert np.array_equal(got, want)
        assert (buf[offset + width * n:] == -7.0).all() and (buf[:offset] == -7.0).all()
    ps.close()


def test_bad_device_values_leave_the_state(gpu):
    import torch
    sc = scenes.pbf_double_dam_break(block=(6, 6, 12))
    ps = rxPBDSPH(sc.params)
    ps.Set(sc.pos, sc.vel)
    ps.Update(sc.dt)
    before = ps.GetArrayVBO(abi.RX_VELOCITY)
    for bad in (float("nan"), float("inf"), -float("inf")):
        t = torch.zeros((sc.n, 4), device="cuda")
        t[sc.n - 1, 2] = bad
        torch.cuda.synchronize()
        assert ps.L.fsph_set_array(ps.handle, abi.RX_VELOCITY, _p(t), 0, sc.n, abi.DEVICE) == abi.NAN_DETECTED
        assert np.array_equal(ps.GetArrayVBO(abi.RX_VELOCITY), before)
    # one of the context's own arrays as the destination
    own = ps.L.fsph_device_ptr(ps.handle, abi.RX_FORCE)
    assert ps.L.fsph_get_array(ps.handle, abi.RX_VELOCITY, ctypes.c_void_p(own), abi.DEVICE, None) == abi.OK
    ps.close()


@pytest.mark.parametrize("offset", [0, 1])
def test_batch_device_arrays(gpu, offset):
    import torch
    scs = scenes.batched_scenes(3, n_lo=100, n_hi=900)
    pos = np.concatenate([s.pos for s in scs])
    b = PBFBatch([s.params for s in scs], [s.n for s in scs], iterations=2)
    buf = torch.zeros(4 * b.n + 8, device="cuda")
    view = buf[offset:offset + 4 * b.n]
    view.copy_(torch.from_numpy(pos.reshape(-1)))
    torch.cuda.synchronize()
    got = []
    for where in (abi.HOST, abi.DEVICE):
        src = pos.ctypes.data_as(ctypes.c_void_p) if where == abi.HOST else _p(view)
        b._check(b._L.fsph_batch_set_particles(b.handle, src, None, where))
        b.step(scs[0].dt)
        got.append([b.get(abi.RX_POSITION), b.get(abi.RX_DENSITY)])
    assert all(np.array_equal(x, y) for x, y in zip(*got))
    for which, width, want in ((abi.RX_POSITION, 4, got[0][0]), (abi.RX_DENSITY, 1, got[0][1])):
        b._check(b._L.fsph_batch_get_array(b.handle, which, _p(view), abi.DEVICE))
        assert np.array_equal(view[:width * b.n].cpu().numpy().reshape(want.shape), want)
    view[5] = float("nan")
    torch.cuda.synchronize()
    assert b._L.fsph_batch_set_particles(b.handle, _p(view), None, abi.DEVICE) == abi.NAN_DETECTED
    b.close()
