"""Phase A's 256-bit loads of an f64 state: a caller's state that is only
16-byte aligned gives the same right-hand side, bit for bit."""

from __future__ import annotations

import ctypes
import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200 import _native as N
from opendynamo_b200.solver import make_params

PREC = {"f64": dict(u_real="f64"), "u64c32": dict(u_real="f64", q_real="f32", rhs_real="f32", compute_real="f32"),
        "mixed": dict(u_real="f64", mixed=True)}


@pytest.mark.gpu
@pytest.mark.parametrize("visc", ["fixed", "sutherland"])
@pytest.mark.parametrize("flux", ["slau2", "ausm+", "rusanov"])
@pytest.mark.parametrize("prec", sorted(PREC))
def test_rhs_of_a_16_byte_aligned_state(prec, flux, visc):
    import torch
    mesh, box = (3, 5, 3), (2 * math.pi, 2.0, math.pi)
    u = torch.from_numpy(np.asarray(channel_trip(*mesh, amp=0.05, dtype=np.float64)).reshape(-1).copy()).cuda()
    p = make_params(*mesh, *box, flux=flux, y_wall=True, viscosity_model=visc, **PREC[prec])
    out = []
    for offset in (0, 2):
        src = torch.zeros(u.numel() + offset, device="cuda", dtype=torch.float64)[offset:]
        src.copy_(u)
        dst = torch.zeros(u.numel() + offset, device="cuda", dtype=torch.float64)[offset:]
        assert src.data_ptr() % 32 == (16 if offset else 0)
        torch.cuda.synchronize()
        rc = N.lib().od_rhs_noalloc(ctypes.byref(p), ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(dst.data_ptr()),
                                    u.numel() * 8, None)
        assert rc == 0
        torch.cuda.synchronize()
        out.append(dst.cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])
    assert np.abs(out[0]).max() > 0
