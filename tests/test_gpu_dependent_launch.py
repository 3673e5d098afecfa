"""Stage kernels launched as programmatic dependents (small meshes): the same
results when the launches are captured and replayed, when copies run between
them, and on both sides of the size where the launches become ordinary ones."""

from __future__ import annotations

import ctypes
import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200 import _native as N
from opendynamo_b200.solver import Solver, make_params

BOX = (2 * math.pi, 2.0, math.pi)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_captured_right_hand_sides_replay(prec):
    import torch
    mesh = (3, 4, 5)
    u = np.asarray(channel_trip(*mesh, amp=0.05, dtype=np.float32 if prec == "f32" else np.float64)).reshape(-1)
    p = make_params(*mesh, *BOX, u_real=prec)
    a = torch.from_numpy(u.copy()).cuda()
    b, c = torch.empty_like(a), torch.empty_like(a)

    def twice(s):   # R(u), then R(R(u)-shifted state): the second reads what the first wrote
        for src, dst in ((a, b), (b, c)):
            rc = N.lib().od_rhs_noalloc(ctypes.byref(p), ctypes.c_void_p(src.data_ptr()),
                                        ctypes.c_void_p(dst.data_ptr()), a.numel() * a.element_size(),
                                        ctypes.c_void_p(s.cuda_stream))
            assert rc == 0
            if dst is b:
                b.mul_(1e-3).add_(a)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        twice(s)
    torch.cuda.synchronize()
    want = (b.cpu().numpy(), c.cpu().numpy())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        twice(s)
    for _ in range(3):
        b.zero_()
        c.zero_()
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(b.cpu().numpy(), want[0])
        np.testing.assert_array_equal(c.cpu().numpy(), want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [(2, 2, 2), (40, 40, 40), (41, 40, 40)])
def test_steps_with_copies_between_them(mesh):
    """(40^3 is below 2^16 elements, 41 x 40 x 40 above.)"""
    import torch
    u = torch.from_numpy(np.asarray(channel_trip(*mesh, amp=0.05, dtype=np.float32)).reshape(-1).copy()).cuda()
    v = torch.empty_like(u)
    torch.cuda.synchronize()
    with Solver(make_params(*mesh, *BOX, u_real="f32")) as s:
        s.set_state_device(u.data_ptr(), s.state_bytes)
        s.step(4, 1e-4)
        s.get_state_device(v.data_ptr(), s.state_bytes)
        s.sync()
        want = v.cpu().numpy()
        # one step at a time, the state out and in again between them
        s.set_state_device(u.data_ptr(), s.state_bytes)
        for _ in range(4):
            s.step(1, 1e-4)
            s.get_state_device(v.data_ptr(), s.state_bytes)
            s.set_state_device(v.data_ptr(), s.state_bytes)
        s.get_state_device(v.data_ptr(), s.state_bytes)
        s.sync()
        np.testing.assert_array_equal(v.cpu().numpy(), want)
    assert np.abs(want - u.cpu().numpy()).max() > 0
