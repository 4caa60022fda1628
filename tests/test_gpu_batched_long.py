"""kv_sweep_batched where two-site vectors are longer than a cluster takes in one Lanczos step, so that a worker's step
is separate launches while a single chain's is one cooperative launch: the same bits either way."""
import numpy as np
import pytest

import kvtest_util as U

U.load_package()
from kylin_v_gb300 import holstein as H  # noqa: E402

pytestmark = pytest.mark.gpu
LONGEST_IN_A_CLUSTER = 77824  # complex elements, on a worker stream


@pytest.fixture(scope="module")
def gpu():
    from kylin_v_gb300 import kvgpu

    kvgpu.init(0)
    return kvgpu


def _longest(mps):
    """Elements of the longest two-site tensor."""
    n = 0
    for x, y in zip(mps[:-1], mps[1:]):
        seen = {(q[0], q[1], r[1], r[2]): a.shape[0] * a.shape[1] * b.shape[1] * b.shape[2]
                for q, a in x.blocks for r, b in y.blocks if q[2] == r[0]}
        n = max(n, sum(seen.values()))
    return n


@pytest.mark.parametrize("prec", [0, 1])
def test_batched_equals_sequential(gpu, prec):
    chains = []
    for seed in (3, 4):
        ch = H.HolsteinChain(3, [0.2, 1.2], [[0.5, 1.0]] * 3, cutoff=12)
        chains.append((H.random_mps(ch, 96, seed=seed), H.hamiltonian_mpo(ch)))
        assert _longest(chains[-1][0]) > LONGEST_IN_A_CLUSTER
    make = lambda: [gpu.TDVP(m, w, 1e-8, 1e-8, 96, 11, 0.05, prec) for m, w in chains]  # noqa: E731
    seq, bat = make(), make()
    for t in seq:
        t.two_site()
    gpu.sweep_batched(bat, 2, 1, max_streams=2)
    for a, b in zip(seq, bat):
        for j in range(a.ns):
            x, y = a.site(j).to_host(), b.site(j).to_host()
            assert [q for q, _ in x.blocks] == [q for q, _ in y.blocks]
            assert all(np.array_equal(u, v) for (_, u), (_, v) in zip(x.blocks, y.blocks)), j
