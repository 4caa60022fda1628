"""Packed tiles of the tensor-core GEMM: many output blocks in one tile, against numpy, exactly.

Small integers are exact in the fixed-point digits and in every accumulation, so whatever the packing does with rows
and columns -- pieces of one row, blocks no multiple of 8, blocks beyond one tile, several segments with and without
shared columns, missing pairs -- the result has to be the integer product, bit for bit."""
import numpy as np
import pytest

import kvtest_util as U

U.load_package()
from kylin_v_gb300.kvio import BlockTensor  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from kylin_v_gb300 import kvgpu

    kvgpu.init(0)
    return kvgpu


def _ints(rng, shape):
    return rng.integers(-9, 10, shape) + 1j * rng.integers(-9, 10, shape)


def _run(gpu, A, B, da, db):
    got = gpu.product(BlockTensor(da, A), BlockTensor(db, B), 1, precision=gpu.KV_MIXED_GEMM).to_host().as_dict()
    want = {}
    for qa, a in A:
        for qb, b in B:
            if qa[-1] == qb[0] and a.shape[-1] == b.shape[0]:
                x = np.tensordot(a, b, 1)
                k = (qa[:-1] + qb[1:], x.shape)
                want[k] = want.get(k, 0) + x
    assert set(got) == set(want)
    for k in want:
        assert np.array_equal(got[k], want[k])


@pytest.mark.parametrize("rows,cols,K", [
    ([8] * 51, [8] * 40, 8), ([1, 2, 3, 5, 7, 9, 11], [1, 3, 8, 17, 31, 32, 33], 5), ([24, 57, 129, 300], [64, 65], 48),
    ([128, 128], [32], 250), ([1], [1], 1), ([40] * 9, [25] * 9, 33), ([136], [200, 7], 16),
])
def test_one_segment_blocks(gpu, rows, cols, K):
    """Every row block meets every column block of its contracted charge (two such charges)."""
    rng = np.random.default_rng([len(rows), len(cols), K])
    A = [((i, q, q), _ints(rng, (m, 1, K + q))) for q in range(2) for i, m in enumerate(rows)]
    B = [((q, q, j), _ints(rng, (K + q, 1, n))) for q in range(2) for j, n in enumerate(cols)]
    _run(gpu, A, B, (1, 1, -1), (1, 1, -1))


@pytest.mark.parametrize("rows,cols,ks,holes", [
    ([8] * 30, [8], [8, 24, 8], False), ([64] * 5, [64], [64, 192, 64], False), ([7, 130, 1], [3, 40], [16, 300], False),
    ([8] * 20, [9, 5], [8, 8, 8, 8], True),
])
def test_several_segments(gpu, rows, cols, ks, holes):
    """Output blocks summing several block pairs; with holes some row blocks lack some of them."""
    rng = np.random.default_rng([len(rows), len(cols), len(ks)])
    A = [((i, s), _ints(rng, (m, k))) for i, m in enumerate(rows) for s, k in enumerate(ks)
         if not (holes and (i + s) % 5 == 0)]
    B = [((s, j), _ints(rng, (k, n))) for s, k in enumerate(ks) for j, n in enumerate(cols)]
    _run(gpu, A, B, (1, -1), (1, -1))
