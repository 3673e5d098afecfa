"""od_diagnostics where its work split has edges: rows of one element, odd
rows (a warp takes two elements), more element rows than blocks fit, fewer
elements than warps, repeated calls on one context."""

from __future__ import annotations

import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200.solver import Solver, make_params
from test_gpu_diag import numpy_diag

BOX = (2 * math.pi, 2.0, math.pi)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mesh", [(1, 1, 1), (1, 3, 1), (3, 2, 5), (9, 1, 11), (2, 450, 1), (13, 4, 17), (40, 2, 30)])
def test_diagnostics_at_the_edges_of_the_split(mesh, prec):
    u = channel_trip(*mesh, amp=0.05, dtype=np.float32 if prec == "f32" else np.float64)
    lx, ly, lz = (float(np.float32(x)) for x in BOX)
    vol, prof = numpy_diag(np.asarray(u), *mesh, lx, ly, lz)
    with Solver(make_params(*mesh, *BOX, "slau2", True, prec)) as s:
        s.set_state(u)
        for _ in range(2):
            d = s.diagnostics()
            got = [d[k] for k in ("mass", "momentum_x", "energy", "kinetic_energy", "enstrophy", "volume")]
            # both sides sum in float64; N terms of one sign (the momentum's wall-bounded
            # profile too) are off by at most about N eps of the sum
            n = mesh[0] * mesh[1] * mesh[2] * 64 + 100
            np.testing.assert_allclose(got, vol, rtol=n * 2.0 ** -52 + 1e-12)
            np.testing.assert_allclose(d["profiles"], prof, rtol=1e-11, atol=n * 2.0 ** -52 * np.abs(prof).max())
        only = s.diagnostics(profiles=False)
        np.testing.assert_allclose([only["mass"], only["enstrophy"]], [vol[0], vol[4]], rtol=n * 2.0 ** -52 + 1e-12)
