"""Kernels launched as programmatic dependents of one another give the bits of
kernels launched one at a time with the host waiting in between, on both sides
of every size where a launch changes from one kind to the other."""

from __future__ import annotations

import math

import numpy as np
import pytest

from helpers import channel_trip
from opendynamo_b200.forms import closure as CL
from opendynamo_b200.slabs import DOWN, UP, Slab
from opendynamo_b200.solver import Solver, make_params
from test_gpu_mlp_fused import run as run_closure

BOX = (2 * math.pi, 2.0, math.pi)
PREC = {"f32": dict(u_real="f32"), "f64": dict(u_real="f64"),
        "u32c64": dict(u_real="f32", q_real="f64", rhs_real="f64", compute_real="f64"),
        "u64c32": dict(u_real="f64", q_real="f32", rhs_real="f32", compute_real="f32"),
        "mixed": dict(u_real="f64", mixed=True)}
# elements: 8, 382 | 384, 639 | 640, 1020 | 1025, 2368 | 2370, 2552 | 2560,
# 3399 | 3400, 4095 | 4096, 65536 | 65600
MESHES = [(2, 2, 2), (2, 191, 1), (8, 8, 6), (9, 71, 1), (10, 8, 8), (17, 12, 5), (5, 5, 41), (37, 8, 8), (6, 5, 79),
          (8, 11, 29), (16, 16, 10), (3, 11, 103), (20, 17, 10), (13, 15, 21), (16, 16, 16), (64, 32, 32), (41, 40, 40)]


def _one_at_a_time(p, u, n_steps, dt):
    """The same steps by one slab that is its own neighbour, the host waiting
    after every kernel and copy."""
    import torch
    s = Slab(p, 0, p.nz)
    try:
        s.set_state(u)
        for _ in range(n_steps):
            for stage in range(3):
                for kind in (0, 1):
                    for d in (DOWN, UP):
                        buf = torch.empty(s.halo_bytes(kind, d), device="cuda", dtype=torch.uint8)
                        s.pack(stage, kind, d, buf)
                        s.sync()
                        s.unpack(stage, kind, d, buf)
                        s.sync()
                    s.stage(stage, kind, dt)
                    s.sync()
        return s.get_state()
    finally:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", MESHES, ids=lambda m: str(m[0] * m[1] * m[2]))
@pytest.mark.parametrize("prec", sorted(PREC))
def test_steps_equal_kernels_run_one_at_a_time(prec, mesh):
    dt = np.float32 if prec in ("f32", "u32c64") else np.float64
    u = np.asarray(channel_trip(*mesh, amp=0.05, dtype=dt)).reshape(-1)
    p = make_params(*mesh, *BOX, flux="slau2", y_wall=True, **PREC[prec])
    want = _one_at_a_time(p, u, 3, 1e-4)
    for epb in (4, 2) if prec != "u32c64" else (4,):
        with Solver(p) as s:
            s.set_state(u)
            s.step(3, 1e-4)
            if epb == 4:
                np.testing.assert_array_equal(s.get_state(), want)
            else:   # another kernel: equal to itself with the host waiting after every step
                s.set_launch_shape(epb, 2)
                s.set_state(u)
                s.step(3, 1e-4)
                got = s.get_state()
                s.set_state(u)
                for _ in range(3):
                    s.step(1, 1e-4)
                    s.sync()
                np.testing.assert_array_equal(s.get_state(), got)
    assert np.abs(want - u).max() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [(13, 15, 21), (16, 16, 16), (5, 8, 13)], ids=lambda m: str(m[0] * m[1] * m[2]))
def test_closure_steps_on_both_sides_of_its_limit(mesh):
    """The fused network after phase A (ordinary below 4096 elements, a
    dependent from there) against the separate features kernel and GEMMs, and
    the same bits from every run."""
    params = CL.init_params(np.random.default_rng(sum(mesh)), out_scale=1.0)
    for k in params:
        if k.startswith("b"):
            params[k] = params[k] + 0.05 * np.random.default_rng(7).standard_normal(params[k].shape).astype(np.float32)
    inc_f, st_f = run_closure(mesh, True, params, 3)
    inc_u, st_u = run_closure(mesh, False, params, 3)
    for _ in range(3):
        np.testing.assert_array_equal(run_closure(mesh, True, params, 3)[1], st_f)
    inc_f, inc_u, st_f, st_u = (x.reshape(5, -1) for x in (inc_f, inc_u, st_f, st_u))
    assert np.all(np.abs(inc_u).max(axis=1) > 1e-4)
    err = np.abs(inc_f - inc_u).max(axis=1) / np.abs(inc_u).max(axis=1)   # bf16 network, as test_gpu_mlp_fused
    assert np.all(err < 1e-4), err
    # 9 stages of f32 round-off: of the state, and of dt times a right-hand side
    # whose largest flux is the pressure, times the Jacobian 2 n / L and the rows
    # of D and g' (absolute sums below 32 together)
    eps, dt = 2.0 ** -24, 2e-4
    p = 0.4 * (st_u[4] - 0.5 * (st_u[1:4] ** 2).sum(axis=0) / st_u[0]).max()
    jac = max(2 * n / l for n, l in zip(mesh, BOX))
    tol = 9 * eps * (np.abs(st_u).max(axis=1) + dt * p * jac * 32)
    assert np.all(np.abs(st_f - st_u).max(axis=1) <= tol)
