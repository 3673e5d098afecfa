"""The closure training step's batch kernels at the edges of their tiles:
batches that end inside a 64-row tile, pools that are not 16-byte aligned,
and every copy of the weights an Adam step writes (row-major, transposed, the
fused inference kernel's image)."""

from __future__ import annotations

import ctypes
import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200 import _native as N
from opendynamo_b200.forms import closure as C
from opendynamo_b200.solver import Solver, make_params


def _pools(rows, offset, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)

    def pool(cols):
        p = torch.empty(rows * cols + offset, device="cuda", dtype=torch.bfloat16)[offset:].view(rows, cols)
        p.copy_(torch.randn(rows, cols, device="cuda", generator=g))
        return p
    return pool(C.N_IN), pool(C.N_OUT)


def _net(params, rows):
    net = C.Network(rows)
    net.set_params(params)
    return net


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("batch", [1, 63, 64, 65, 129, 1000])
def test_train_step_is_one_adam_step_on_the_batch_gradient(batch, offset):
    import torch
    X, T = _pools(batch + 37, offset, batch)
    rows = np.random.default_rng(batch).permutation(batch + 37)[:batch].astype(np.int64)
    p0 = C.init_params(np.random.default_rng(3))
    net = _net(p0, batch)
    loss = net.train_step(X, T, rows, 1e-3)
    got = net.get_params()
    # the same batch gathered here
    M = (batch + 127) // 128 * 128
    at = torch.from_numpy(rows).cuda()
    Xb = torch.zeros(M, C.N_IN, device="cuda", dtype=torch.bfloat16)
    Xb[:batch] = X[at]
    Tb = torch.zeros(M, C.N_OUT_PAD, device="cuda")
    Tb[:batch, :C.N_OUT] = T[at].float()
    grads, want_loss = _net(p0, batch).gradients(Xb, Xb.t().contiguous(), Tb, batch)
    assert abs(loss - want_loss) <= 1e-12 * want_loss   # the same float squares, summed in float64
    for k, g in grads.items():
        g = g.astype(np.float64)
        m, v = 0.1 * g, 0.001 * g * g
        step = 1e-3 * (m / 0.1) / (np.sqrt(v / 0.001) + 1e-8)
        # the step is at most 1e-3; a dozen f32 roundings on its way (the bias
        # corrections 1 - 0.999 lose up to 2^-24 / 1e-3 of themselves), then the
        # rounding of the weight
        tol = 1e-3 * (12 * 2.0 ** -24 + 2.0 ** -24 / 1e-3) + 2.0 ** -23 * np.abs(p0[k])
        assert np.all(np.abs(got[k] - (p0[k] - step)) <= tol), k


@pytest.mark.gpu
def test_every_copy_of_the_weights_follows_the_step():
    import torch
    X, T = _pools(256, 0, 1)
    net = _net(C.init_params(np.random.default_rng(5)), 256)
    for k in range(2):
        net.train_step(X, T, np.arange(256), 1e-2)
    fresh = _net(net.get_params(), 256)
    Tb = torch.zeros(256, C.N_OUT_PAD, device="cuda")
    # forward (W) and backward (W^T)
    a, la = net.gradients(X, X.t().contiguous(), Tb, 256)
    b, lb = fresh.gradients(X, X.t().contiguous(), Tb, 256)
    assert abs(la - lb) <= 1e-12 * lb
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    # the fused inference image: a solver step with the closure attached
    n, box = 4, (2 * math.pi, 2.0, math.pi)
    u = channel_trip(n, n, n, amp=0.05, dtype=np.float32)
    out = []
    for m in (net, fresh):
        m.set_scaling(np.zeros(14), np.ones(14), np.full(5, 0.1))
        with Solver(make_params(n, n, n, *box, "slau2", True, "f32")) as s:
            s.set_state(u)
            m.attach(s)
            s.step(2, 1e-3)
            out.append(s.get_state())
            C.Network.detach(s)
    np.testing.assert_array_equal(out[0], out[1])
    assert np.abs(out[0] - u).max() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("M,N_,K", [(128, 64, 64), (256, 192, 320), (256, 896, 4096)])
def test_gemm_output_alignment(M, N_, K, offset):
    """Products with and without split K into 16-byte aligned and other buffers."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(K)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N_, K, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(N_, device="cuda", generator=g)
    out = torch.zeros(M * N_ + offset, device="cuda")[offset:]
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())   # noqa: E731
    assert N.lib().od_gemm_bf16(M, N_, K, p(A), p(B), p(out), p(bias), None) == 0
    torch.cuda.synchronize()
    want = A.double() @ B.double().T + bias.double()
    size = A.double().abs() @ B.double().abs().T + bias.double().abs()
    # f32 accumulation of K exact products in any order
    assert torch.all((out.view(M, N_).double() - want).abs() <= (K + 2) * 2.0 ** -24 * size)
