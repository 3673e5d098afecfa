"""od_set_state_device and od_get_state_device copy: they take any address the
copy takes, also one that no kernel could read as the state's type."""

from __future__ import annotations

import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200.solver import Solver, make_params

BOX = (2 * math.pi, 2.0, math.pi)
MESH = (3, 2, 3)
PREC = {"f32": dict(u_real="f32"), "f64": dict(u_real="f64"),
        "u64c32": dict(u_real="f64", q_real="f32", rhs_real="f32", compute_real="f32"),
        "mixed": dict(u_real="f64", mixed=True)}


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [1, 4, 8, 12])
@pytest.mark.parametrize("prec", sorted(PREC))
def test_state_at_a_byte_offset(prec, offset):
    import torch
    dt = np.float32 if prec == "f32" else np.float64
    u = np.asarray(channel_trip(*MESH, amp=0.05, dtype=np.float64)).reshape(-1)
    u = (u * (1 + 1e-9 * np.random.default_rng(0).standard_normal(u.size))).astype(dt)
    raw = torch.from_numpy(u.view(np.uint8).copy())
    src = torch.zeros(raw.numel() + offset, device="cuda", dtype=torch.uint8)[offset:]
    dst = torch.zeros(raw.numel() + offset, device="cuda", dtype=torch.uint8)[offset:]
    src.copy_(raw)
    torch.cuda.synchronize()

    def got(s):
        dst.zero_()
        torch.cuda.synchronize()
        s.get_state_device(dst.data_ptr(), u.nbytes)
        s.sync()
        return dst.cpu().numpy().view(dt)

    with Solver(make_params(*MESH, *BOX, **PREC[prec])) as s:
        s.set_state(u)
        s.step(2, 1e-3)
        want = s.get_state()
        s.set_state_device(src.data_ptr(), u.nbytes)
        np.testing.assert_array_equal(got(s), u)
        np.testing.assert_array_equal(s.get_state(), u)
        s.step(2, 1e-3)
        np.testing.assert_array_equal(got(s), want)
        np.testing.assert_array_equal(s.get_state(), want)
