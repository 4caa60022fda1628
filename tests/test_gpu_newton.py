"""The FP64 SVD's reciprocal and reciprocal square root (two Newton steps on an FP32 start, csrc/kv_rotation64.cuh)
against CUDA's own division and square root and against extended precision, and the rotation it builds from them.

Two Newton steps leave an error of the start's, at most 2^-21, to the fourth power, and the last one rounds twice: two
units in the last place are allowed.  CUDA's quotient 1 / x is half a unit from the exact one, 1 / sqrt(x) one and a
half, so the two forms may differ by three and a half.  A rotation is unitary to 8 x 2^-53 whatever its angle, and its
angle, from 24-bit mantissas, leaves less than 1e-5 of the pair's cosine."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import kvtest_util as U

U.load_package()
from kylin_v_gb300 import build as B  # noqa: E402

pytestmark = pytest.mark.gpu

SRC = """
#include "kv_rotation64.cuh"
using namespace kv::rot64;
__global__ void k(const double *x, int n, double *o) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        o[i] = newton_reciprocal(x[i]);
        o[n + i] = 1.0 / x[i];
        o[2 * n + i] = newton_rsqrt(x[i]);
        o[3 * n + i] = 1.0 / sqrt(x[i]);
    }
}
__global__ void kr(const double *x, int n, double *o) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        rotation(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3], o[3 * i], o[3 * i + 1], o[3 * i + 2]);
}
static int run(const double *x, int nx, int n, double *o, int no, bool rot) {
    double *dx, *dout;
    if (cudaMalloc(&dx, nx * 8) || cudaMalloc(&dout, no * 8)) return 1;
    if (cudaMemcpy(dx, x, nx * 8, cudaMemcpyHostToDevice)) return 2;
    if (rot) kr<<<64, 128>>>(dx, n, dout);
    else k<<<64, 128>>>(dx, n, dout);
    if (cudaMemcpy(o, dout, no * 8, cudaMemcpyDeviceToHost)) return 3;
    return (int)cudaFree(dx) + (int)cudaFree(dout);
}
extern "C" int newton(const double *x, int n, double *o) { return run(x, n, n, o, 4 * n, false); }
extern "C" int rotations(const double *x, int n, double *o) { return run(x, 4 * n, n, o, 3 * n, true); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("newton")
    (d / "n.cu").write_text(SRC)
    so = str(d / "n.so")
    subprocess.run([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", B.CSRC,
                    str(d / "n.cu"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _call(f, x, n, no):
    x, o = np.ascontiguousarray(x), np.empty(no)
    p = ctypes.POINTER(ctypes.c_double)
    assert f(x.ctypes.data_as(p), n, o.ctypes.data_as(p)) == 0
    return o


def _inputs():
    rng = np.random.default_rng(1)
    near = np.concatenate([np.nextafter(2.0**np.arange(-40, 41), d) for d in (0, 1, 1e300)])
    return np.concatenate([2.0 ** rng.uniform(-860, 860, 200000), rng.uniform(1, 4, 200000), near,
                           2.0**np.arange(-860, 861.0)])


def test_reciprocal_and_root(lib):
    x = _inputs()
    rec, div, rsq, root = _call(lib.newton, x, len(x), 4 * len(x)).reshape(4, -1)
    assert np.array_equal(div, 1.0 / x)
    if np.finfo(np.longdouble).nmant > 60:
        xl = x.astype(np.longdouble)
        for got, want in ((rec, 1 / xl), (rsq, 1 / np.sqrt(xl))):
            assert (np.abs(got - want) / np.spacing(want.astype(float))).max() <= 2
    assert (np.abs(rec - div) / np.spacing(div)).max() <= 2.5
    assert (np.abs(rsq - root) / np.spacing(root)).max() <= 3.5


def test_rotation(lib):
    """[[a, c], [c*, b]] with |c| <= sqrt(a b) over the range of squared column norms."""
    rng = np.random.default_rng(2)
    n = 200000
    a, b = 10.0 ** rng.uniform(-260, 6, n), None
    b = np.where(rng.random(n) < 0.5, a * 10.0 ** rng.uniform(-3, 3, n), 10.0 ** rng.uniform(-260, 6, n))
    b = np.where(rng.random(n) < 0.1, a, np.clip(b, 1e-260, 1e7))
    c = np.sqrt(a) * np.sqrt(b) * 10.0 ** rng.uniform(-15, 0, n) * np.exp(2j * np.pi * rng.random(n))
    o = _call(lib.rotations, np.stack([a, b, c.real, c.imag], 1), n, 3 * n).reshape(n, 3)
    cs, s = o[:, 0], o[:, 1] + 1j * o[:, 2]
    assert np.abs(cs**2 + np.abs(s) ** 2 - 1).max() <= 8 * 2.0**-53
    # the cosine left: x' = cs x - conj(s) y, y' = s x + cs y, in units of sqrt(a b) (scaled so that b <= a = 1)
    u = np.sqrt(np.minimum(a, b) / np.maximum(a, b))
    big = a >= b
    aa, bb = np.where(big, 1.0, u**2), np.where(big, u**2, 1.0)
    cc = c / np.maximum(a, b)
    # <x', y'> = cs s a + cs^2 c - s^2 conj(c) - cs s b, with s^2 conj(c) = |s|^2 c
    left = cs * s * (aa - bb) + (cs**2 - np.abs(s) ** 2) * cc
    assert (np.abs(left) / np.abs(cc)).max() <= 1e-5
