"""The block permutation's index arithmetic (csrc/kv_permute.cuh) compiled for the host, against numpy: every
permutation of every rank, unit lengths among the axes, both index widths, and blocks of more than 2^31 elements at
sampled elements."""
import ctypes
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

import kvtest_util as U

SRC = """
#include "kv_permute.cuh"
extern "C" void perm(const int64_t *shape, const int64_t *axes, int rank, int64_t n, const int64_t *e, int wide,
                     int64_t *out) {
    const kvp::PermMap m = kvp::perm_map(shape, axes, rank);
    for (int64_t i = 0; i < n; ++i) out[i] = kvp::perm_index(m, rank, e[i], wide != 0);
}
"""


@pytest.fixture(scope="module")
def perm(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ absent")
    d = tmp_path_factory.mktemp("perm")
    (d / "p.cpp").write_text(SRC)
    so = str(d / "p.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-fPIC", "-shared", "-I",
                    os.path.join(U.ROOT, "kylin-v_gb300", "csrc"), str(d / "p.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def call(shape, axes, e, wide):
        arr = [np.ascontiguousarray(x, dtype=np.int64) for x in (shape, axes, e)]
        out = np.empty(len(arr[2]), np.int64)
        p = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)) for a in (*arr, out)]
        lib.perm(p[0], p[1], len(shape), ctypes.c_int64(len(out)), p[2], int(wide), p[3])
        return out

    return call


@pytest.mark.parametrize("shape", [(1,), (7,), (3, 5), (1, 4), (2, 1, 3), (4, 3, 2, 5), (3, 1, 2, 1, 4),
                                   (2, 3, 1, 4, 2, 3)])
def test_every_permutation(perm, shape):
    n = int(np.prod(shape))
    for axes in itertools.permutations(range(len(shape))):
        # element e goes to the place where the transposed array holds e
        want = np.argsort(np.arange(n).reshape(shape).transpose(axes).ravel())
        for wide in (False, True):
            assert np.array_equal(perm(shape, axes, np.arange(n), wide), want), (axes, wide)


@pytest.mark.parametrize("shape", [(70000, 65537), (3, 5, 1 << 28), (1 << 16, 3, 1 << 15, 7), (2, 1 << 30, 3)])
def test_large_blocks(perm, shape):
    rng = np.random.default_rng(len(shape))
    n = int(np.prod(shape, dtype=object))
    assert n >= 1 << 31
    e = np.concatenate([rng.integers(0, n, 1000), [0, n - 1, (1 << 31) - 1, 1 << 31]])
    for axes in itertools.permutations(range(len(shape))):
        idx = np.unravel_index(e, shape)
        strides = [int(np.prod([shape[a] for a in axes[j + 1:]], dtype=object)) for j in range(len(axes))]
        want = sum(idx[a].astype(np.int64) * strides[j] for j, a in enumerate(axes))
        assert np.array_equal(perm(shape, axes, e, True), want), axes
