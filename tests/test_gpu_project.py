"""od_project at every factor, type combination and pointer alignment, on
coarse meshes whose element count is no multiple of the block's, against the
L2 projection in float64."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from opendynamo_b200 import _native as N


def projection_matrix(f):
    """P[i, a]: coarse node i from the fine sample a of a row of f elements."""
    xi, w = np.polynomial.legendre.leggauss(4)
    P = np.zeros((4, 4 * f))
    for a in range(4 * f):
        x = -1.0 + (2.0 * (a // 4) + 1.0 + xi[a % 4]) / f
        for i in range(4):
            lag = np.prod([(x - xi[m]) / (xi[i] - xi[m]) for m in range(4) if m != i])
            P[i, a] = w[a % 4] * lag / (f * w[i])
    return P


def project64(u, n, f, P):
    nx, ny, nz = n
    t = u.reshape(5, nz, f, ny, f, nx, f, 4, 4, 4).transpose(0, 1, 3, 5, 2, 7, 4, 8, 6, 9)
    t = t.reshape(5, nz, ny, nx, 4 * f, 4 * f, 4 * f)   # (c, b, a) fine samples of a coarse element
    return np.einsum("kc,jb,ia,vzyxcba->vzyxkji", P, P, P, t, optimize=True).reshape(5, -1)


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("types", [(np.float32, np.float32), (np.float64, np.float32), (np.float32, np.float64),
                                   (np.float64, np.float64)])
@pytest.mark.parametrize("factor", range(1, 9))
def test_projection_matches_float64(factor, types, offset):
    import torch
    n = (3, 1, 2) if factor > 4 else (3, 5, 2)
    ne = n[0] * n[1] * n[2]
    rng = np.random.default_rng(factor)
    u = rng.standard_normal(5 * ne * factor ** 3 * 64).astype(types[0])
    td = {np.float32: torch.float32, np.float64: torch.float64}
    src = torch.zeros(u.size + offset, device="cuda", dtype=td[types[0]])[offset:]
    src.copy_(torch.from_numpy(u))
    dst = torch.zeros(5 * ne * 64 + offset, device="cuda", dtype=td[types[1]])[offset:]
    torch.cuda.synchronize()
    rc = N.lib().od_project(ctypes.c_void_p(src.data_ptr()), int(types[0] is np.float64), *n, factor,
                            ctypes.c_void_p(dst.data_ptr()), int(types[1] is np.float64), None)
    assert rc == 0
    torch.cuda.synchronize()
    got = dst.cpu().numpy().astype(np.float64).reshape(5, -1)
    P = projection_matrix(factor)
    want = project64(u.astype(np.float64), n, factor, P)
    # three f32 sums of 4 f products each, three rounded table entries, one rounded input
    size = project64(np.abs(u).astype(np.float64), n, factor, np.abs(P))
    assert np.all(np.abs(got - want) <= (3 * 4 * factor + 4) * 2.0 ** -24 * size)
