"""The mixed SVD with a sector on a cluster of CTAs: the shapes where dealing the reduction's rows and the Jacobi's
columns can go wrong (the smallest sector that gets a cluster, row counts that do not divide, more rows than one pass
holds, wide rows that leave no room for the exchange, rank-deficient sectors that end the reduction early).

The row updates and rotations are the same arithmetic wherever they run, so the result must equal, bit for bit, that
of the same sector among so many others that each gets one CTA.  Against the matrix itself: values below 1e-6 of the
largest count as zero and FP32 chooses the subspace, so U V is allowed 1e-5 of the largest singular value; the kept
factor comes from an FP64 Cholesky-QR pass on columns orthonormal to FP32 rounding: 1e-12."""
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


def _split(gpu, mats, l2r):
    t = BlockTensor((1, -1), [((q, q), a) for q, a in enumerate(mats)])
    L, R, _, _ = gpu.svd_impl(t, 1, l2r, 0.0, sum(min(a.shape) for a in mats), precision=gpu.KV_MIXED_TF32)
    return {q[0]: a for q, a in L.to_host().blocks}, {q[1]: a for q, a in R.to_host().blocks}


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("rank", [None, 3, 37])
@pytest.mark.parametrize("m,n", [(32, 32), (33, 65), (64, 64), (65, 33), (67, 67), (127, 128), (128, 127), (128, 128),
                                 (40, 150), (150, 40), (90, 300)])
def test_cluster_equals_one_cta(gpu, m, n, rank, l2r):
    rng = np.random.default_rng([m, n, rank or 0])
    a = rng.normal(size=(m, n)) + 1j * rng.normal(size=(m, n))
    if rank is not None:
        k = min(rank, m, n)
        a = (rng.normal(size=(m, k)) + 1j * rng.normal(size=(m, k))) @ a[:k]
    L, R = _split(gpu, [a], l2r)
    L1, R1 = _split(gpu, [a] + [np.full((1, 1), 1.0 + q) for q in range(159)], l2r)
    assert np.array_equal(L[0], L1[0]) and np.array_equal(R[0], R1[0])
    s0 = np.linalg.svd(a, compute_uv=False)[0]
    assert np.abs(L[0] @ R[0] - a).max() <= 1e-5 * s0
    x = L[0] if l2r else R[0].conj().T
    assert np.abs(x.conj().T @ x - np.eye(x.shape[1])).max() <= 1e-12
