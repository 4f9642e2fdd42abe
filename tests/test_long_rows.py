"""Draws where a node's rows are too long to stage, and where the buffer sets are
so large that a launch draws two iterations."""
import numpy as np
import pytest

import oracle
from mcmc_for_ammsb_gb300 import MCMCSamplerStochastic, Network, Options

pytestmark = pytest.mark.gpu


# a hub of 300 links (256 are staged) and 40 held-out partners (32 are), and one
# past every staging area of the minibatch kernel too: neighbour sets exactly
# those of the oracle
@pytest.mark.parametrize("links,partners", [(256, 32), (300, 33), (3000, 700)])
def test_neighbour_sets_of_a_hub(native_lib, links, partners):
    N, n_out, steps = 5000, 41, 40
    rng = np.random.default_rng(links)
    others = rng.permutation(np.arange(1, N))
    a, b = rng.integers(1, N, 10000), rng.integers(1, N, 10000)
    net = Network.from_edges(N, np.concatenate([a, np.zeros(links, np.int64)]), np.concatenate([b, others[:links]]))
    net.held_out = (np.zeros(partners, np.int32), others[links:links + partners].astype(np.int32),
                    np.zeros(partners, np.uint8))
    net.test = (np.array([1], np.int32), np.array([2], np.int32), np.zeros(1, np.uint8))
    s = MCMCSamplerStochastic(Options(K=4, num_node_sample=n_out - 1, mini_batch_size=2000, strategy=2), net).init()
    og, hubs = oracle.OracleGraph(net), 0
    for step in range(1, steps + 1):
        s.step(1)
        mb = s.last_minibatch()
        for r in np.flatnonzero(mb["nodes"] == 0).tolist() + [0, 1000, 2000]:
            nb, y = oracle.sample_neighbors(og, int(mb["nodes"][r]), n_out, 42, 0, step)
            assert np.array_equal(mb["nbrs"][r], nb) and np.array_equal(mb["nbr_y"][r], y)
            hubs += mb["nodes"][r] == 0
    assert hubs > 3


# 20,000 nodes x 1,001 neighbour words are 80 MB a buffer set: blocks of two
def test_large_buffer_sets_take_blocks_of_two(native_lib):
    rng = np.random.default_rng(2)
    N = 20000
    net = Network.from_edges(N, rng.integers(0, N, 60000), rng.integers(0, N, 60000))
    net.make_held_out(0.01, seed=2)
    opts = dict(K=4, num_node_sample=1000, mini_batch_size=20000, strategy=3)
    states = []
    for pipeline, pieces in ((1, (1, 4, 2, 5)), (0, (12,))):
        s = MCMCSamplerStochastic(Options(pipeline=pipeline, **opts), net).init()
        for n in pieces:
            s.step(n)
        states.append([s.phi, s.theta, s.last_minibatch()["nbrs"]])
        s.close()
    for x, y in zip(*states):
        assert np.array_equal(x, y)
