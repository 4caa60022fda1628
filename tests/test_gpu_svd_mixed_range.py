"""The mixed SVD of sectors with a few rows or columns of about 1e-20 beside ordinary ones (in FP32 the squares of such
entries are subnormal): the reflectors of the reduction must stay unitary, in shared memory on one CTA and on a
cluster, and beyond shared memory.

Tolerances: the kept factor is rebuilt from the FP32 vectors of the other side, whose pairs are orthogonal to 1e-5 (the
rotation tolerance), an error that enters the singular values squared, once per other state: n 1e-10 of the largest
value; the kept factor itself is a Cholesky-QR of columns orthonormal to FP32: 1e-12; U V is the projection of the
sector on the states kept, of which those below 1e-6 of the largest count as zero: 1e-5."""
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


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("power", [-17, -18, -19, -20, -20.5, -21, -21.5, -22, -22.3, -24, -40])
@pytest.mark.parametrize("m,n,faint", [(40, 30, 1), (40, 30, 20), (20, 25, 3), (128, 100, 30), (260, 200, 60)])
def test_faint_rows_and_columns(gpu, m, n, faint, power, l2r):
    rng = np.random.default_rng([m, n, faint])
    a = rng.normal(size=(m, n)) + 1j * rng.normal(size=(m, n))
    a[:, :faint] *= 10.0**power
    for z in (a, a.T.copy()):
        L, R, k, _ = gpu.svd_impl(BlockTensor((1, -1), [((0, 0), z)]), 1, l2r, 0.0, n,
                                  precision=gpu.KV_MIXED_TF32)
        x, y = L.to_host().blocks[0][1], R.to_host().blocks[0][1]
        s = np.linalg.svd(z, compute_uv=False)
        orth, other = (x, y) if l2r else (y.conj().T, x.T)
        assert np.abs(orth.conj().T @ orth - np.eye(k)).max() <= 1e-12
        assert np.abs(x @ y - z).max() <= 1e-5 * s[0]
        assert np.abs(np.linalg.norm(other, axis=1) - s[:k]).max() <= max(m, n) * 1e-10 * s[0]


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("m,n", [(64, 64), (64, 90), (65, 65), (66, 100), (100, 65)])
def test_either_side_of_the_cluster_rule(gpu, m, n, l2r):
    """64 columns take one CTA, 65 a cluster: the bits of the same sector among so many that each gets one CTA."""
    rng = np.random.default_rng([m, n])
    a = rng.normal(size=(m, n)) + 1j * rng.normal(size=(m, n))
    out = []
    for others in (0, 159):
        mats = [a] + [np.full((1, 1), 1.0 + q) for q in range(others)]
        t = BlockTensor((1, -1), [((q, q), x) for q, x in enumerate(mats)])
        L, R, _, _ = gpu.svd_impl(t, 1, l2r, 0.0, min(m, n) + others, precision=gpu.KV_MIXED_TF32)
        out.append((dict(L.to_host().blocks)[(0, 0)], dict(R.to_host().blocks)[(0, 0)]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    x, y = out[0]
    assert np.abs(x @ y - a).max() <= 1e-5 * np.linalg.svd(a, compute_uv=False)[0]
