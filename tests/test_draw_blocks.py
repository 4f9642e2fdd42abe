"""The draws of a block of iterations made by one launch, on the GPU: a chain
stepped in pieces that start, end and cross blocks anywhere is the chain
stepped in the loop's order, bit for bit."""
import numpy as np
import pytest

from mcmc_for_ammsb_gb300 import ChainBatch, MCMCSamplerStochastic, Options, _native, workloads

pytestmark = pytest.mark.gpu

PIECES = [1, 1, 6, 3, 16, 5, 8, 2, 13, 7, 24, 1]  # 87 iterations


@pytest.fixture(scope="module")
def net(native_lib):
    return workloads.build("diff")[0]


def state(s):
    mb = s.last_minibatch()
    return [s.phi, s.pi, s.theta, s.beta, mb["nodes"], mb["nbrs"], np.int64(s.step_count),
            np.array(s.counters())]


@pytest.fixture(scope="module")
def in_order(net):
    s = MCMCSamplerStochastic(Options(K=16, num_node_sample=32, pipeline=0), net).init()
    s.step(sum(PIECES))
    return state(s)


@pytest.mark.parametrize("graph", [1, 0])
@pytest.mark.parametrize("block", ["1", "2", "3", "8", "16"])
def test_pieces_give_the_same_chain(net, in_order, monkeypatch, block, graph):
    monkeypatch.setenv("AMMSB_GRAPH_PAIRS", block)
    s = MCMCSamplerStochastic(Options(K=16, num_node_sample=32, use_graph=graph), net).init()
    for i, n in enumerate(PIECES):
        s.step(n)
        if i == 4:  # the draws made ahead are dropped and made again
            s.set_step(s.step_count)
    for a, b in zip(state(s), in_order):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("iters", ["2", "6", "16"])
def test_batch_pieces_give_the_same_chain(net, in_order, monkeypatch, iters):
    monkeypatch.setenv("AMMSB_BATCH_GRAPH_ITERS", iters)
    chains = [MCMCSamplerStochastic(Options(K=16, num_node_sample=32, pi_dtype=_native.PI_F32,
                                            chain=c), net).init() for c in (0, 1)]
    batch = ChainBatch(chains)
    for i, n in enumerate(PIECES):
        if i == 6:  # on its own in between: the batch draws again
            chains[0].step(n)
            chains[1].step(n)
        else:
            batch.step(n)
    for a, b in zip(state(chains[0]), in_order):
        assert np.array_equal(a, b)
