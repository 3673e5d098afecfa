"""The arithmetic of the f64 pipelines on the device: division and reciprocal
are correctly rounded under either math policy (as numpy's are), also for
zeros, infinities and subnormals; the precision form's refined reciprocal is
within its bound for both f32 estimates it starts from."""

from __future__ import annotations

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "od_physics.cuh"
using namespace od;
__global__ void ops(const double* a, const double* b, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = MathIeee::rcp(b[i]);
    out[n + i] = MathIeee::div(a[i], b[i]);
    out[2 * n + i] = MathFast::rcp(b[i]);
    out[3 * n + i] = MathFast::div(a[i], b[i]);
    out[4 * n + i] = rcp_refined(b[i], MathIeee::rcp((float)b[i]));
    out[5 * n + i] = rcp_refined(b[i], MathFast::rcp((float)b[i]));
}
extern "C" int run(const double* a, const double* b, double* out, int n) {
    double *da, *db, *dout;
    const size_t s = sizeof(double) * n;
    if (cudaMalloc(&da, s) || cudaMalloc(&db, s) || cudaMalloc(&dout, 6 * s)) return 1;
    if (cudaMemcpy(da, a, s, cudaMemcpyHostToDevice) || cudaMemcpy(db, b, s, cudaMemcpyHostToDevice)) return 2;
    ops<<<(n + 127) / 128, 128>>>(da, db, dout, n);
    if (cudaGetLastError() || cudaMemcpy(out, dout, 6 * s, cudaMemcpyDeviceToHost)) return 3;
    return cudaFree(da) || cudaFree(db) || cudaFree(dout);
}
"""


@pytest.fixture(scope="module")
def run_ops(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("ops")
    src, lib = str(d / "ops.cu"), str(d / "libops.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I" + os.path.join(ROOT, "opendynamo_b200", "csrc"), "-o", lib, src], check=True)
    fn = ctypes.CDLL(lib).run

    def call(a, b):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        out = np.empty((6, a.size))
        p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, out)]
        assert fn(*p, a.size) == 0
        return out

    return call


def _mantissas(rng, n):
    m = rng.uniform(1.0, 2.0, n)
    return np.concatenate([m, 1.0 + np.arange(64) * 2.0 ** -52, 2.0 - np.arange(1, 65) * 2.0 ** -52])


@pytest.mark.gpu
def test_division_is_correctly_rounded(run_ops):
    rng = np.random.default_rng(0)
    b = _mantissas(rng, 200000)
    b = b * 2.0 ** rng.integers(-300, 300, b.size) * rng.choice([-1.0, 1.0], b.size)
    a = rng.permutation(b)
    tiny, huge = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, tiny, -tiny, tiny / 2, 5e-324, -5e-324, huge, -huge, 1.0, -3.0])
    sa, sb = (x.reshape(-1) for x in np.meshgrid(special, special))
    a, b = np.concatenate([a, sa]), np.concatenate([b, sb])
    out = run_ops(a, b)
    with np.errstate(all="ignore"):
        rcp, quo = 1.0 / b, a / b
    for got, want in ((out[0], rcp), (out[1], quo), (out[2], rcp), (out[3], quo)):
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(np.signbit(got[want == 0]), np.signbit(want[want == 0]))


@pytest.mark.gpu
def test_refined_reciprocal_of_the_f32_estimates(run_ops):
    """The estimates are within 2^-22 (an f32 rounding of the operand, 2^-24, and
    at most an ulp, 2^-23, of the result), so that e^3 is below 2^-66 and the
    result is off by half an ulp for its own rounding and at most 2^-12 ulp."""
    rng = np.random.default_rng(1)
    x = _mantissas(rng, 200000)
    x = x * 2.0 ** rng.integers(-100, 100, x.size)
    out = run_ops(x, x)
    assert np.finfo(np.longdouble).nmant >= 63
    xl = x.astype(np.longdouble)
    exact = 1 / xl                                     # within 2^-64: 2^-12 ulp of an f64 more at most
    ulp = np.spacing((1.0 / x)).astype(np.longdouble)
    for got in (out[4], out[5]):
        assert (np.abs(got - exact) / ulp).max() <= 0.5 + 2.0 ** -11
