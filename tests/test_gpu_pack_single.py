"""Tensor-core GEMM plans of blocks that pack with no other: each pair of operand blocks has a contracted charge of its
own.  Runs of equal blocks (which share their tiles' row and column maps), alternating sizes, single rows, and blocks of
exactly and just over one tile (128 rows, 32 columns), against numpy on small integers, exactly."""
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


@pytest.mark.parametrize("sizes", [
    [(8, 8, 8)] * 200, [(8, 8, 8), (8, 16, 8), (16, 8, 8)] * 9, [(1, 1, 1)] * 5 + [(2, 1, 300)] * 3,
    [(128, 32, 16), (129, 32, 16), (128, 33, 16), (32, 32, 16), (40, 32, 16)] * 2, [(5, 7, 3), (130, 70, 250), (5, 7, 3)],
])
def test_lone_blocks(gpu, sizes):
    rng = np.random.default_rng([len(sizes), *sizes[0]])
    ints = lambda *s: rng.integers(-9, 10, s) + 1j * rng.integers(-9, 10, s)  # noqa: E731
    A = [((i, i), ints(m, k)) for i, (m, n, k) in enumerate(sizes)]
    B = [((i, i), ints(k, n)) for i, (m, n, k) in enumerate(sizes)]
    got = dict(gpu.product(BlockTensor((1, -1), A), BlockTensor((1, -1), B), 1,
                           precision=gpu.KV_MIXED_GEMM).to_host().blocks)
    assert len(got) == len(sizes)
    for (q, a), (_, b) in zip(A, B):
        assert np.array_equal(got[q], a @ b)
