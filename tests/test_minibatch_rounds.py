"""Non-link minibatches past 4,096, drawn eight at once, against the oracle's
sequential scan: rounds of more candidates than the minibatch has edges, a
dedup hash in shared memory and in per-iteration areas of global memory, and a
source whose links and held-out partners are too many to stage."""
import numpy as np
import pytest

import oracle
from mcmc_for_ammsb_gb300 import MCMCSamplerStochastic, Network, Options

pytestmark = pytest.mark.gpu

N, STEPS, HUB_STEP = 60000, 18, 11  # three blocks of draws; the hub is the source of one


@pytest.fixture(scope="module")
def net(native_lib):
    rng = np.random.default_rng(1)
    a, b = rng.integers(0, N, 120000), rng.integers(0, N, 120000)
    plain = Network.from_edges(N, a, b)
    plain.held_out = plain.test = (np.array([0], np.int32), np.array([1], np.int32), np.zeros(1, np.uint8))
    hub = oracle.sample_minibatch(oracle.OracleGraph(plain), 2, 8, plain.num_total_edges, 42, 0, HUB_STEP,
                                  64)["nodes"][0]
    others = rng.permutation(np.delete(np.arange(N), hub))
    net = Network.from_edges(N, np.concatenate([a, np.full(3000, hub)]), np.concatenate([b, others[:3000]]))
    partners = others[3000:3700].astype(np.int32)
    net.held_out = (np.full(700, hub, np.int32), partners, np.zeros(700, np.uint8))
    net.test = (others[:50].astype(np.int32), others[50:100].astype(np.int32), np.zeros(50, np.uint8))
    return net


@pytest.mark.parametrize("m", [4096, 4097, 5000, 8193, 10000])
def test_large_minibatches_are_the_sequential_scan(net, m):
    opts = dict(K=4, num_node_sample=4, mini_batch_size=m, strategy=2, random_seed=42)
    s = MCMCSamplerStochastic(Options(**opts), net).init()
    og = oracle.OracleGraph(net)
    for step in range(1, STEPS + 1):
        s.step(1)
        got = s.last_minibatch()
        want = oracle.sample_minibatch(og, 2, m, net.num_total_edges, 42, 0, step, s.max_edges)
        for k in ("edge_a", "edge_b", "edge_y", "nodes"):
            assert np.array_equal(got[k], want[k]), (step, k)
    in_order = MCMCSamplerStochastic(Options(pipeline=0, **opts), net).init()
    in_order.step(STEPS)
    for name in ("phi", "pi", "theta"):
        assert np.array_equal(getattr(s, name), getattr(in_order, name)), name
