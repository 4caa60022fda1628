"""The MPO mixing kernel where an output block sums several input blocks: as many terms as a warp's list holds and more,
terms of different contracted lengths, dense and sparse lists that fit and that do not, and row lengths on each side of
the kernel's three walks -- an H_eff apply whose environments are identities, against numpy.

Input block i has left charge -i, physical charge i and the MPO bond's charge i, so every one of them reaches the one
output block of charges 0: y[a, s', b] = sum_i sum_{w, s, v} W_i[s', w, s, v] psi_i[a, s, b].  Sums of n products:
8 (n + 4) 2^-53 n max|W| max|psi| is allowed."""
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


@pytest.mark.parametrize("kind", ["complex", "sparse", "unit"])
@pytest.mark.parametrize("b", [1, 16, 17, 33, 64, 65, 130])
@pytest.mark.parametrize("terms,so,wr", [(2, 3, 2), (2, 1, 1), (16, 1, 1), (16, 2, 3), (17, 1, 1), (40, 2, 2)])
def test_terms_of_one_block(gpu, terms, so, wr, b, kind):
    rng = np.random.default_rng([terms, so, wr, b])
    a = 7
    L, p, m = [], [], []
    for i in range(terms):
        wl, d = 1 + i % 2, 1 + i % 3  # contracted lengths 1, 4, 3, 2, 2, 6
        W = rng.normal(size=(so, wl, d, wr)) + 1j * rng.normal(size=(so, wl, d, wr))
        if kind == "sparse":
            W = np.where(rng.random(W.shape) < 0.1, W, 0)
        if kind == "unit":
            W = np.where(rng.random(W.shape) < 0.2, 1.0, 0) + 0j
        L.append(((0, i, -i), np.repeat(np.eye(a)[:, None, :], wl, 1) + 0j))
        p.append(((-i, i, 0), rng.normal(size=(a, d, b)) + 1j * rng.normal(size=(a, d, b))))
        m.append(((0, i, i, 0), W))
    # every (left, site) pair of charges that meets an MPO block feeds output block (0, 0, 0)
    feeds = [1 for (_, w, x), _ in L for (y, s, _), _ in p for (_, w2, s2, _), _ in m if x == y and (w, s) == (w2, s2)]
    assert len(feeds) == terms
    want = sum(np.einsum("swtv,atb->asb", W, x) for (_, W), (_, x) in zip(m, p))
    R = BlockTensor((-1, 1, 1), [((0, 0, 0), np.repeat(np.eye(b)[:, None, :], wr, 1) + 0j)])
    got = gpu.heff_apply(1, BlockTensor((1, -1, -1), L), BlockTensor((1, 1, -1), p), BlockTensor((1, 1, -1, -1), m),
                         None, R).to_host()
    got = dict(got.blocks)
    y = got.pop((0, 0, 0))
    assert not any(x.any() for x in got.values())  # psi's other blocks: zeros
    n = wr * sum(W.shape[1] * W.shape[2] for _, W in m)
    big = max(1e-300, max(np.abs(W).max() for _, W in m)) * max(np.abs(x).max() for _, x in p)
    assert np.abs(y - want).max() <= 8 * (n + 4) * 2.0**-53 * n * big
