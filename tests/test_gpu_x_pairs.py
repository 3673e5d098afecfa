"""Elements that share a warp exchange their traces at a common x face; the
others read them. A periodic shift by one element along x changes which do, and
the result shifts with the state, bit for bit, whatever the row length."""

from __future__ import annotations

import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200.solver import Solver, make_params

BOX = (2 * math.pi, 2.0, math.pi)
PREC = {"f32": dict(u_real="f32"), "f64": dict(u_real="f64"),
        "u64c32": dict(u_real="f64", q_real="f32", rhs_real="f32", compute_real="f32"),
        "mixed": dict(u_real="f64", mixed=True)}


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("prec", sorted(PREC))
def test_a_shift_along_x_shifts_the_result(prec, nx):
    mesh = (nx, 2, 3)
    p = make_params(*mesh, *BOX, flux="slau2", y_wall=True, **PREC[prec])
    dt = np.float32 if prec == "f32" else np.float64
    rng = np.random.default_rng(nx)
    u = np.asarray(channel_trip(*mesh, amp=0.05, dtype=np.float64)).reshape(5, 3, 2, nx, 64)
    u = (u * (1 + 1e-3 * rng.standard_normal(u.shape))).astype(dt)
    out = []
    for shift in (0, 1):
        with Solver(p) as s:
            s.set_state(np.roll(u, shift, axis=3).reshape(-1))
            s.step(2, 1e-4)
            out.append(np.roll(s.get_state().reshape(u.shape), -shift, axis=3))
    assert np.isfinite(out[0]).all() and np.abs(out[0] - u).max() > 0
    np.testing.assert_array_equal(out[0], out[1])
