"""od_diagnostics of a state with infinite values: the sums that hold them are
infinite, as the sum of their terms is, wherever the element lies in its row (a
warp takes two elements of a row; the last may have no partner)."""

from __future__ import annotations

import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200.solver import Solver, make_params

BOX = (2 * math.pi, 2.0, math.pi)


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [(1, 1, 1), (3, 2, 3), (2, 2, 2)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_an_infinite_energy_stays_in_its_sum(prec, mesh):
    dt = np.float32 if prec == "f32" else np.float64
    u = np.asarray(channel_trip(*mesh, amp=0.05, dtype=dt)).copy()
    with Solver(make_params(*mesh, *BOX, "slau2", True, prec)) as s:
        s.set_state(u)
        clean = s.diagnostics()
        u.reshape(5, -1)[4, -1] = np.inf   # the last point of the last element of the last row
        s.set_state(u)
        d = s.diagnostics()
    assert d["energy"] == np.inf
    for k in ("mass", "momentum_x", "kinetic_energy", "enstrophy", "volume"):
        assert d[k] == pytest.approx(clean[k], rel=1e-11, abs=1e-11)
    np.testing.assert_allclose(d["profiles"], clean["profiles"], rtol=1e-11, atol=1e-13)


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [(1, 1, 1), (3, 2, 3), (2, 2, 2)])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_an_infinite_density_stays_in_the_mass(prec, mesh):
    dt = np.float32 if prec == "f32" else np.float64
    u = np.asarray(channel_trip(*mesh, amp=0.05, dtype=dt)).copy()
    u.reshape(5, -1)[0, -1] = np.inf
    with Solver(make_params(*mesh, *BOX, "slau2", True, prec)) as s:
        s.set_state(u)
        d = s.diagnostics()
    assert d["mass"] == np.inf
    assert d["profiles"].reshape(-1, 8)[-1, 0] == np.inf
