"""The FP64 block SVD against numpy, sector by sector, at the shapes where its split can go wrong: single rows and
columns, wide and tall sectors, every register width and the streamed form (more than 256 rows), cluster sizes from
one CTA up, odd ranks, rank-deficient and zero sectors, strongly graded and repeated singular values.

Tolerances: one-sided Jacobi and the Householder reduction are backward stable with a bound of a modest multiple of
n 2^-53 |A| (n the larger side); 40 n 2^-53 |A|_2 is allowed for singular values and for U S V^H, and the kept factor
is orthonormal to the rotation tolerance 1e-15 per pair plus rounding: 1e-14 + 40 n 2^-53 per entry."""
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


def _matrix(rng, m, n, kind):
    a = rng.normal(size=(m, n)) + 1j * rng.normal(size=(m, n))
    k = min(m, n)
    if kind == "random":
        return a
    if kind == "zero":
        return 0 * a
    if kind == "zerorows":  # exactly zero rows and columns
        a[m // 2:] = 0
        a[:, n // 2:] = 0
        return a
    u, _, v = np.linalg.svd(a, full_matrices=False)
    s = {"rank": np.where(np.arange(k) < max(1, k // 3), 1.0, 0.0) * np.linspace(1, 0.5, k),
         "graded": 10.0 ** (-30.0 * np.arange(k) / max(1, k - 1)),
         "repeated": np.where(np.arange(k) < k // 2, 1.0, 1e-3)}[kind]
    return (u * s) @ v


def _check(gpu, mats, l2r):
    t = BlockTensor((1, -1), [((q, q), a) for q, a in enumerate(mats)])
    kmax = sum(min(a.shape) for a in mats)
    L, R, kept, total = gpu.svd_impl(t, 1, l2r, -1.0, kmax)  # nothing truncated
    assert total == kmax and kept == kmax
    L, R = {q[0]: a for q, a in L.to_host().blocks}, {q[1]: a for q, a in R.to_host().blocks}
    for q, a in enumerate(mats):
        n = max(a.shape)
        x, y = L[q], R[q]
        s = np.linalg.svd(a, compute_uv=False)
        tol = 40 * n * EPS * s[0]
        assert np.abs(x @ y - a).max() <= tol
        orth, other = (x, y) if l2r else (y.conj().T, x.conj().T)
        k = orth.shape[1]
        assert np.abs(orth.conj().T @ orth - np.eye(k)).max() <= 1e-14 + 40 * n * EPS
        got = np.linalg.norm(other, axis=1)  # the other factor's rows carry the singular values
        assert np.abs(got - s).max() <= tol


@pytest.mark.parametrize("l2r", [True, False])
@pytest.mark.parametrize("kind", ["random", "rank", "graded", "repeated", "zerorows", "zero"])
@pytest.mark.parametrize("shapes", [
    [(1, 1)], [(1, 9), (9, 1)], [(2, 3), (3, 2), (5, 5)], [(64, 64), (65, 63)], [(101, 101)] * 3,
    [(128, 40), (40, 128)], [(129, 77)], [(256, 33)], [(300, 50), (50, 300)], [(7, 2000)], [(16, 16)] * 40,
])
def test_sectors(gpu, shapes, kind, l2r):
    rng = np.random.default_rng([len(shapes), shapes[0][0], shapes[0][1]])
    _check(gpu, [_matrix(rng, m, n, kind) for m, n in shapes], l2r)


def test_long_pivot_row(gpu):
    """A sector wider than the staged pivot row (4096 columns)."""
    rng = np.random.default_rng(5)
    _check(gpu, [_matrix(rng, 12, 4501, "random")], True)


def test_non_finite(gpu):
    rng = np.random.default_rng(6)
    a = _matrix(rng, 20, 20, "random")
    a[3, 4] = np.nan
    t = BlockTensor((1, -1), [((0, 0), a), ((1, 1), _matrix(rng, 8, 8, "random"))])
    with pytest.raises(gpu.KvError):
        gpu.svd_impl(t, 1, True, 1e-8, 8)
    _check(gpu, [_matrix(rng, 20, 20, "random")], True)
