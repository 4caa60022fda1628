"""The MPO mixing kernel at the edges of its per-warp lists: more terms, outputs or nonzero entries than a list holds,
single elements, chunk boundaries, complex, real, unit and zero MPO entries -- an H_eff apply and an environment
update whose environments are identities, against numpy.

With L and R the identity the apply is the mixing itself: y[a, s', b] = sum_s W[s', 1, s, 1] psi[a, s, b], and with an
MPO bond of dimension w (L[a', w, a] = R[b', w, b] = delta at every w) the sum over both bond indices.  Sums of n
products: 8 (n + 4) 2^-53 n max|W| max|psi| is allowed."""
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


def _mpo(rng, d, w, kind):
    W = rng.normal(size=(d, w, d, w)) + 1j * rng.normal(size=(d, w, d, w))
    if kind == "real":
        W = W.real + 0j
    if kind == "sparse":
        W = np.where(rng.random(W.shape) < 0.2, W.real, 0) + 0j
    if kind == "unit":
        W = np.einsum("st,uv->sutv", np.eye(d), np.eye(w)) + 0j
    if kind == "zero":
        W = 0 * W
    return W


@pytest.mark.parametrize("kind", ["complex", "real", "sparse", "unit", "zero"])
@pytest.mark.parametrize("d,w,a,b,sectors", [
    (1, 1, 1, 1, False), (2, 3, 5, 7, False), (4, 4, 3, 1, False), (5, 4, 2, 31, False), (3, 9, 4, 33, False),
    (20, 1, 2, 3, True), (17, 2, 5, 9, True), (2, 2, 64, 65, True), (3, 2, 130, 70, False),
])
def test_apply_is_the_mixing(gpu, d, w, a, b, sectors, kind):
    rng = np.random.default_rng([d, w, a, b])
    W = _mpo(rng, d, w, kind)
    psi = rng.normal(size=(a, d, b)) + 1j * rng.normal(size=(a, d, b))
    eye = lambda n: np.repeat(np.eye(n)[:, None, :], w, 1) + 0j  # noqa: E731
    L, R = BlockTensor((1, -1, -1), [((0, 0, 0), eye(a))]), BlockTensor((-1, 1, 1), [((0, 0, 0), eye(b))])
    if sectors:  # physical states as blocks of their own (all of charge 0 but distinguished by shape is not possible,
        # so they get charges s, and the bond on the right too): one term per input state
        p = BlockTensor((1, 1, -1), [((0, s, s), psi[:, s:s + 1]) for s in range(d)])
        m = BlockTensor((1, 1, -1, -1), [((s, 0, s, 0), W[s:s + 1, :, s:s + 1]) for s in range(d)])
        R = BlockTensor((-1, 1, 1), [((s, 0, s), eye(b)) for s in range(d)])
        want = {(0, s, s): np.einsum("wv,ab->ab", W[s, :, s], psi[:, s])[:, None] for s in range(d)}
    else:
        p, m = BlockTensor((1, 1, -1), [((0, 0, 0), psi)]), BlockTensor((1, 1, -1, -1), [((0, 0, 0, 0), W)])
        want = {(0, 0, 0): np.einsum("swtv,atb->asb", W, psi)}
    got = {q: x for q, x in gpu.heff_apply(1, L, p, m, None, R).to_host().blocks}
    n = d * w * w
    tol = 8 * (n + 4) * 2.0**-53 * n * max(1e-300, np.abs(W).max()) * np.abs(psi).max()
    for q, x in want.items():
        assert np.abs(got[q] - x).max() <= tol
