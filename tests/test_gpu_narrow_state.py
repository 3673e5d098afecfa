"""The u64/c32 pipeline holds its state in f32 between calls (its state
arithmetic is f32, so every stored value is one). Against the paths that
store f64: a slab decomposition and the context-free right-hand side, bit for
bit; and the caller's f64 state comes back untouched until a step."""

from __future__ import annotations

import ctypes
import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200 import _native as N
from opendynamo_b200.slabs import LocalSlabs
from opendynamo_b200.solver import Solver, make_params

BOX = (2 * math.pi, 2.0, math.pi)
PREC = dict(u_real="f64", q_real="f32", rhs_real="f32", compute_real="f32")
MESH = (5, 3, 4)


def _params(flux="slau2", wall=True, visc="fixed", **kw):
    return make_params(*MESH, *BOX, flux=flux, y_wall=wall, viscosity_model=visc, **PREC, **kw)


def _state(seed=0):
    """f64 values that are no f32 values."""
    u = np.asarray(channel_trip(*MESH, amp=0.05, dtype=np.float64)).reshape(-1)
    return u * (1 + 1e-9 * np.random.default_rng(seed).standard_normal(u.size))


@pytest.mark.gpu
@pytest.mark.parametrize("fast_math", [True, False])
@pytest.mark.parametrize("visc", ["fixed", "sutherland"])
@pytest.mark.parametrize("flux,wall", [("slau2", True), ("ausm+", False), ("rusanov", True)])
def test_steps_equal_the_f64_storage(flux, wall, visc, fast_math):
    p = _params(flux, wall, visc, fast_math=fast_math)
    u = _state()
    d = LocalSlabs(p, 2)
    try:
        d.set_state(u)
        d.step(5, 1e-3)
        want = d.get_state()
    finally:
        d.close()
    with Solver(p) as s:
        s.set_state(u)
        s.step(5, 1e-3)
        got = s.get_state()
        np.testing.assert_array_equal(got, want)
        # a state that went out and in again goes on the same
        s.step(3, 1e-3)
        far = s.get_state()
        s.set_state(got)
        s.step(3, 1e-3)
        np.testing.assert_array_equal(s.get_state(), far)


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
def test_the_callers_state_is_kept_until_a_step(offset):
    import torch
    u, v = _state(1), _state(2)
    with Solver(_params()) as s:
        s.set_state(u)
        np.testing.assert_array_equal(s.get_state(), u)
        mass = s.diagnostics()["mass"]
        s.step(0, 1e-3)
        np.testing.assert_array_equal(s.get_state(), u)
        # device copies, of any alignment
        src = torch.zeros(u.size + offset, device="cuda", dtype=torch.float64)[offset:]
        dst = torch.zeros(u.size + offset, device="cuda", dtype=torch.float64)[offset:]
        src.copy_(torch.from_numpy(v))
        torch.cuda.synchronize()
        s.set_state_device(src.data_ptr(), u.nbytes)
        s.get_state_device(dst.data_ptr(), u.nbytes)
        s.sync()
        np.testing.assert_array_equal(dst.cpu().numpy(), v)
        s.step(2, 1e-3)
        want = s.get_state()
        s.set_state_device(src.data_ptr(), u.nbytes)
        s.step(2, 1e-3)
        s.get_state_device(dst.data_ptr(), u.nbytes)
        s.sync()
        np.testing.assert_array_equal(dst.cpu().numpy(), want)
        np.testing.assert_array_equal(want, want.astype(np.float32).astype(np.float64))
    with Solver(make_params(*MESH, *BOX, u_real="f64")) as s:   # the f64 pipeline's sum of the same state
        s.set_state(u)
        assert s.diagnostics()["mass"] == pytest.approx(mass, rel=1e-14)


@pytest.mark.gpu
def test_asynchronous_transfers_and_right_hand_side():
    import torch
    u = _state(3)
    p = _params()
    stream = torch.cuda.Stream()
    host = torch.from_numpy(u.copy()).pin_memory()
    back = torch.empty_like(host).pin_memory()
    with Solver(p) as s:
        s.set_state(u)
        s.step(4, 1e-3)
        want = s.get_state()
        L = N.lib()
        assert L.od_set_state_async(s._ctx, ctypes.c_void_p(host.data_ptr()), u.nbytes,
                                    ctypes.c_void_p(stream.cuda_stream)) == 0
        s.step(4, 1e-3)
        assert L.od_get_state_async(s._ctx, ctypes.c_void_p(back.data_ptr()), u.nbytes,
                                    ctypes.c_void_p(stream.cuda_stream)) == 0
        s.step(2, 1e-3)   # must not reach the download
        stream.synchronize()
        np.testing.assert_array_equal(back.numpy(), want)
        s.set_state(u)
        got = s.rhs()
        np.testing.assert_array_equal(s.get_state(), u)   # a right-hand side leaves the state alone
    a = torch.from_numpy(u).cuda()
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    assert N.lib().od_rhs_noalloc(ctypes.byref(p), ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()),
                                  u.nbytes, None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(got, b.cpu().numpy())
