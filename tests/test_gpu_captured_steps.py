"""Steps and state copies captured on a context's stream and replayed: the
state that the calls after a replay see is the one the replay left, also for
the u64/c32 pipeline, whose caller's view of the state is kept apart from the
stored one."""

from __future__ import annotations

import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200.solver import Solver, make_params

BOX = (2 * math.pi, 2.0, math.pi)
MESH = (5, 3, 4)
PREC = {"f32": dict(u_real="f32"), "f64": dict(u_real="f64"),
        "u64c32": dict(u_real="f64", q_real="f32", rhs_real="f32", compute_real="f32"),
        "mixed": dict(u_real="f64", mixed=True)}


def _state(prec, seed):
    """Values that are no f32 values where the state is f64."""
    u = np.asarray(channel_trip(*MESH, amp=0.05, dtype=np.float64)).reshape(-1)
    u = u * (1 + 1e-9 * np.random.default_rng(seed).standard_normal(u.size))
    return u.astype(np.float32 if prec == "f32" else np.float64)


def _eager(p, u, n):
    """The state after 1 .. n steps, and the mass and momentum of each."""
    out = []
    with Solver(p) as s:
        s.set_state(u)
        for _ in range(n):
            s.step(1, 1e-3)
            d = s.diagnostics()
            out.append((s.get_state(), d["mass"], d["kinetic_energy"]))
    return out


def _same(s, want):
    d = s.diagnostics()
    # f64 sums in an order that varies: N terms are off by at most about N eps
    assert d["mass"] == pytest.approx(want[1], rel=1e-11)
    assert d["kinetic_energy"] == pytest.approx(want[2], rel=1e-11)
    np.testing.assert_array_equal(s.get_state(), want[0])


@pytest.mark.gpu
@pytest.mark.parametrize("prec", sorted(PREC))
def test_replayed_steps(prec):
    import torch
    p = make_params(*MESH, *BOX, flux="slau2", y_wall=True, **PREC[prec])
    u, v = _state(prec, 1), _state(prec, 2)
    want_u, want_v = _eager(p, u, 3), _eager(p, v, 1)
    with Solver(p) as s:
        ext = torch.cuda.ExternalStream(s.stream)
        s.set_state(u)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=ext):
            s.step(1, 1e-3)
        np.testing.assert_array_equal(s.get_state(), u)   # nothing has run yet

        def replay():
            with torch.cuda.stream(ext):
                g.replay()

        for k in range(2):
            replay()
            _same(s, want_u[k])
        s.step(1, 1e-3)   # enqueued and replayed steps mix
        _same(s, want_u[2])
        s.set_state(v)
        np.testing.assert_array_equal(s.get_state(), v)
        replay()
        _same(s, want_v[0])
        s.set_state(u)
        s.step(1, 1e-3)
        replay()
        _same(s, want_u[1])
        del g


@pytest.mark.gpu
@pytest.mark.parametrize("prec", sorted(PREC))
def test_replayed_state_copies(prec):
    import torch
    p = make_params(*MESH, *BOX, flux="slau2", y_wall=True, **PREC[prec])
    u, v = _state(prec, 3), _state(prec, 4)
    want_u, want_v = _eager(p, u, 2), _eager(p, v, 1)
    src, dst = torch.from_numpy(v).cuda(), torch.zeros(v.size, device="cuda", dtype=torch.from_numpy(v).dtype)
    torch.cuda.synchronize()

    def capture(*calls):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=ext):
            for c in calls:
                c()
        return g

    def replay(g):
        with torch.cuda.stream(ext):
            g.replay()
        s.sync()
        return dst.cpu().numpy()

    with Solver(p) as s:
        ext = torch.cuda.ExternalStream(s.stream)
        put = lambda: s.set_state_device(src.data_ptr(), v.nbytes)   # noqa: E731
        get = lambda: s.get_state_device(dst.data_ptr(), v.nbytes)   # noqa: E731
        step = lambda: s.step(1, 1e-3)                               # noqa: E731
        s.set_state(u)
        g_get, g_put, g_step_get = capture(get), capture(put), capture(step, get)
        np.testing.assert_array_equal(s.get_state(), u)
        np.testing.assert_array_equal(replay(g_get), u)
        s.step(1, 1e-3)
        np.testing.assert_array_equal(replay(g_get), want_u[0][0])
        np.testing.assert_array_equal(replay(g_step_get), want_u[1][0])
        replay(g_put)
        np.testing.assert_array_equal(s.get_state(), v)
        np.testing.assert_array_equal(replay(g_get), v)
        np.testing.assert_array_equal(replay(g_step_get), want_v[0][0])
        _same(s, want_v[0])
        del g_get, g_put, g_step_get
