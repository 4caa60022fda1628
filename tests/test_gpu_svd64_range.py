"""The FP64 block SVD at the ends of the FP64 range: sectors whose squares overflow or underflow, rows so short that the
inner products of two of them underflow or that they count as zero beside the others.

Tolerances as for the SVD of ordinary sectors: 40 n 2^-53 |A|_2 (n the larger side) for singular values and U S V^H,
1e-14 + 40 n 2^-53 per entry for the kept factor's orthonormality; rows below 1e-130 of the largest element may be
dropped, which is far below both."""
import numpy as np
import pytest

import kvtest_util as U

U.load_package()
from kylin_v_gb300.kvio import BlockTensor  # noqa: E402

pytestmark = pytest.mark.gpu
EPS = 2.0**-53


@pytest.fixture(scope="module")
def gpu():
    from kylin_v_gb300 import kvgpu

    kvgpu.init(0)
    return kvgpu


def _random(rng, m, n):
    return rng.normal(size=(m, n)) + 1j * rng.normal(size=(m, n))


def _check(gpu, a, l2r, scale=1.0):
    """The split of a * scale (a itself of ordinary size)."""
    k = min(a.shape)
    L, R, kept, total = gpu.svd_impl(BlockTensor((1, -1), [((0, 0), a * scale)]), 1, l2r, -1.0, k)
    assert kept == total == k
    x, y = L.to_host().blocks[0][1], R.to_host().blocks[0][1]
    x, y = (x, y / scale) if l2r else (x / scale, y)
    n = max(a.shape)
    s = np.linalg.svd(a, compute_uv=False)
    tol = 40 * n * EPS * s[0]
    assert np.abs(x @ y - a).max() <= tol
    orth, other = (x, y) if l2r else (y.conj().T, x.conj().T)
    assert np.abs(orth.conj().T @ orth - np.eye(k)).max() <= 1e-14 + 40 * n * EPS
    assert np.abs(np.linalg.norm(other, axis=1) - s).max() <= tol


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("power", [-300, -165, -158, -155, -150, -100, 150, 160, 300])
@pytest.mark.parametrize("m,n", [(6, 5), (5, 6), (70, 65), (130, 20)])
def test_whole_sector(gpu, m, n, power, l2r):
    _check(gpu, _random(np.random.default_rng([m, n]), m, n), l2r, 10.0**power)


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("power", [-60, -100, -125, -129, -130, -131, -140, -150, -155, -158, -165, -300])
@pytest.mark.parametrize("m,n,short", [(20, 20, 5), (7, 30, 3), (90, 70, 40), (70, 90, 69)])
def test_short_rows(gpu, m, n, short, power, l2r):
    rng = np.random.default_rng([m, n, short])
    a = _random(rng, m, n)
    a[m - short:] *= 10.0**power
    _check(gpu, a, l2r)
    _check(gpu, a.T.copy(), l2r)


@pytest.mark.parametrize("l2r", [True, False])
def test_graded_to_the_floor(gpu, l2r):
    """Rows at every decade from 1 to 1e-320."""
    a = _random(np.random.default_rng(3), 65, 40) * 10.0 ** (-5.0 * np.arange(65))[:, None]
    _check(gpu, a, l2r)


@pytest.mark.parametrize("power", [-155, -158])
def test_a_faint_sector_beside_another(gpu, power):
    """One sector of small amplitude does not fail the split of the others."""
    rng = np.random.default_rng(4)
    a, b = _random(rng, 9, 8), _random(rng, 6, 5) * 10.0**power
    L, R, kept, total = gpu.svd_impl(BlockTensor((1, -1), [((0, 0), a), ((1, 1), b)]), 1, True, 1e-8, 13)
    assert (kept, total) == (8, 13)
    x, y = dict(L.to_host().blocks)[(0, 0)], dict(R.to_host().blocks)[(0, 0)]
    assert np.abs(x @ y - a).max() <= 40 * 9 * EPS * np.linalg.svd(a, compute_uv=False)[0]


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("power", [-140, -149, -150, -151, -155, -158, -159, -160, -161, -161.5, -161.8, -163, -310])
@pytest.mark.parametrize("m,n,at", [(6, 5, 0), (5, 6, 0), (20, 30, 7), (30, 20, 19), (9, 1, 0)])
def test_faint_column(gpu, m, n, at, power, l2r):
    """A column of entries whose squares are subnormal beside ordinary ones: the reflectors' phases."""
    a = _random(np.random.default_rng([m, n]), m, n)
    a[:, at] *= 10.0**power
    if n == 1:
        a[0, 0] = 1.0
    _check(gpu, a, l2r)
    _check(gpu, a.T.copy(), l2r)


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("m,n,rows", [(1, 1, 0), (5, 5, 0), (5, 9, 2), (9, 5, 4), (33, 70, 31), (70, 33, 20),
                                      (300, 40, 39), (260, 270, 1), (100, 100, 50)])
def test_completed_vectors(gpu, m, n, rows, l2r):
    """All min(m, n) states kept of a sector of which only `rows` rows are not zero, and several such sectors."""
    rng = np.random.default_rng([m, n, rows])
    a = np.zeros((m, n), complex)
    a[rng.permutation(m)[:rows]] = _random(rng, rows, n)
    if not a.any():
        k = min(m, n)
        L, R, kept, _ = gpu.svd_impl(BlockTensor((1, -1), [((0, 0), a)]), 1, l2r, -1.0, k)
        x, y = L.to_host().blocks[0][1], R.to_host().blocks[0][1]
        orth, other = (x, y) if l2r else (y.conj().T, x)
        assert kept == k and not other.any()
        assert np.abs(orth.conj().T @ orth - np.eye(k)).max() <= 1e-14 + 40 * max(m, n) * EPS
        return
    _check(gpu, a, l2r)
    _check(gpu, a.T.copy(), l2r)


def test_dropped_vectors_cost_nothing(gpu):
    """A sector of zeros whose states the truncation drops takes no longer than one of full rank."""
    import time

    import torch

    def run(a):
        t, best = gpu.Tensor.from_host(BlockTensor((1, -1), [((0, 0), a)])), 1e9
        for _ in range(4):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            gpu.svd_impl(t, 1, True, 0.0, 200)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        return best

    full = run(_random(np.random.default_rng(8), 200, 200))
    assert run(np.zeros((200, 200), complex)) <= full
