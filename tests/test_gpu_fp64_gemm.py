"""The FP64 grouped GEMM's tiles and K slices against numpy, at the sizes where the split can go wrong:
single elements, blocks no tile divides, K shorter than the number of slices, one output with a very long K,
several segments per output, and the operand forms N / C and N / T.

Tolerance: a sum of n products computed in any order differs from the exact one by at most
(n + 4) 2^-53 sum |a||b| to first order (complex: four real products per term), bounded here by
8 (n + 4) 2^-53 n max|a| max|b|."""
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


def _rand(rng, shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


@pytest.mark.parametrize("m,n,ks", [
    (1, 1, [1]), (1, 3, [7, 4999]), (2, 2, [300]), (3, 5, [1, 2, 3]), (16, 16, [17]), (17, 16, [16, 1]),
    (57, 31, [33, 5, 64]), (64, 200, [8]), (255, 1, [40, 40]), (300, 257, [129]), (8, 8, [2] * 70),
])
@pytest.mark.parametrize("form", ["NN", "CN", "NT"])
def test_product_blocks(gpu, m, n, ks, form):
    rng = np.random.default_rng([m, n, len(ks)])
    # one output block, one segment per contracted charge q (block q of A meets block q of B)
    A = [((0, q), _rand(rng, (m, k))) for q, k in enumerate(ks)]
    B = [((q, 0), _rand(rng, (k, n))) for q, k in enumerate(ks)]
    want = sum(a @ b for (_, a), (_, b) in zip(A, B))
    opA = opB = gpu.OP_N
    a, b = BlockTensor((1, -1), A), BlockTensor((1, -1), B)
    if form == "CN":  # op C: the conjugate, contracted over its first leg
        a = BlockTensor((-1, 1), [((q, 0), x.conj().T.copy()) for (_, q), x in A])
        a = BlockTensor((-1, 1), a.blocks)
        b = BlockTensor((-1, 1), B)
        opA = gpu.OP_C
    if form == "NT":
        b = BlockTensor((-1, 1), [((0, q), x.T.copy()) for (q, _), x in B])
        opB = gpu.OP_T
    got = gpu.product(a, b, 1, opA, opB).to_host()
    assert len(got.blocks) == 1
    big = max(np.abs(x).max() for _, x in A) * max(np.abs(x).max() for _, x in B)
    k = sum(ks)
    assert np.abs(got.blocks[0][1] - want).max() <= 8 * (k + 4) * 2.0**-53 * k * big
