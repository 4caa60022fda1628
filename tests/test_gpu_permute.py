"""The block permutation on the device, through a right-to-left environment update (it permutes the site tensor by
(2, 1, 0) and the MPO tensor by (0, 3, 2, 1)): blocks of less than, exactly and more than one CTA's chunk of 1024
elements, many blocks of different sizes in one launch, a block that spreads over the chip.

The update is sum A*[x, s, b] W[s, w, t, v] env[b, v, c] A[y, t, c]; sums of n products:
8 (n + 4) 2^-53 n max|W| max|env| max|A|^2 is allowed."""
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


def _random(rng, shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


@pytest.mark.parametrize("shapes", [
    [(1, 1, 1)], [(3, 5, 7)], [(8, 4, 32)], [(25, 41, 1)], [(1, 3, 683)], [(31, 3, 11), (1, 1, 1), (40, 6, 9)],
    [(2, 1 + i % 3, 1 + i % 5) for i in range(60)], [(96, 12, 96)],
])
def test_right_to_left(gpu, shapes):
    rng = np.random.default_rng([len(shapes), *shapes[0]])
    # block i of A: left and right charge i, site charge 0; the MPO: one block of charges 0
    d = shapes[0][1]
    shapes = [(a, d, b) for a, _, b in shapes]
    A = [((i, 0, i), _random(rng, s)) for i, s in enumerate(shapes)]
    W = _random(rng, (d, 3, d, 2))
    env = [((i, 0, i), _random(rng, (s[2], 2, s[2]))) for i, s in enumerate(shapes)]
    out = gpu.env_sweep(BlockTensor((-1, 1, 1), env), BlockTensor((1, 1, -1), A),
                        BlockTensor((1, 1, -1, -1), [((0, 0, 0, 0), W)]), False).to_host()
    got = {q: x for q, x in out.blocks}
    assert len(got) == len(shapes)
    for i, (a, _, b) in enumerate(shapes):
        x, e = A[i][1], env[i][1]
        t = np.tensordot(e, x, ([2], [2]))  # [b, v, y, t]
        t = np.tensordot(W, t, ([2, 3], [3, 1]))  # [s, w, b, y]
        want = np.tensordot(x.conj(), t, ([1, 2], [0, 2]))  # [x, w, y]
        n = d * d * 2 * b * b
        big = np.abs(W).max() * np.abs(x).max() ** 2 * np.abs(e).max()
        match = [y for q, y in got.items() if q[0] == i and q[2] == i]
        assert len(match) == 1
        assert np.abs(match[0] - want).max() <= 8 * (n + 4) * 2.0**-53 * n * big
