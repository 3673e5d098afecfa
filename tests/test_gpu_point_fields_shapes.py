"""od_point_fields where its work split has edges: odd and single elements
along z (a warp takes eight), fewer elements than a block's warps, buffers
that are not 16-byte aligned; bit for bit against the conversion script's
arithmetic."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from opendynamo_b200 import _native as N
from oracle import pointfields as PF


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("mesh", [(1, 1, 1), (1, 2, 3), (5, 1, 2), (2, 3, 17), (7, 5, 9)])
def test_point_fields_at_the_edges(mesh, dtype, offset):
    import torch
    n = mesh[0] * mesh[1] * mesh[2] * 64
    rng = np.random.default_rng(n)
    a = rng.standard_normal((5, n)).astype(dtype)
    a[0, ::7] = 0.0
    a[0, 1::11] = np.nan
    d = torch.zeros(a.size + offset, device="cuda", dtype=torch.from_numpy(a).dtype)[offset:]
    d.copy_(torch.from_numpy(a.reshape(-1)))
    out = torch.zeros(7 * n + offset, device="cuda")[offset:]
    torch.cuda.synchronize()
    rc = N.lib().od_point_fields(ctypes.c_void_p(d.data_ptr()), int(dtype is np.float64), *mesh,
                                 ctypes.c_void_p(out.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(7, -1)
    with np.errstate(all="ignore"):
        want = PF.point_fields(a, *mesh)
    for k, name in enumerate(PF.FIELD_NAMES):
        np.testing.assert_array_equal(got[k], np.asarray(want[name], np.float32).reshape(-1), err_msg=name)
