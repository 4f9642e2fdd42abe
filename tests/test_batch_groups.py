"""Batches of chains whose commits are of several kinds -- one edge per summing
warp at once, four, and general edge lists -- and whose update_phi takes a launch
per kind of iteration: bit for bit the chains stepped alone."""
import numpy as np
import pytest

from mcmc_for_ammsb_gb300 import ChainBatch, MCMCSamplerStochastic, Network, Options, _native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(native_lib):
    net = Network.synthetic(n=5000, k_true=50, intra_degree=6.0, seed=9)
    net.make_held_out(0.02, seed=9)
    return net


def check(net, kinds, steps=(5, 16, 3)):
    opts = [Options(num_node_sample=8, chain=c, **kw) for c, kw in enumerate(kinds)]
    alone = [MCMCSamplerStochastic(o, net).init() for o in opts]
    together = [MCMCSamplerStochastic(o, net).init() for o in opts]
    batch = ChainBatch(together)
    for n in steps:
        batch.step(n)
        for s in alone:
            s.step(n)
    for a, b in zip(alone, together):
        for name in ("phi", "pi", "theta", "beta"):
            assert np.array_equal(getattr(a, name), getattr(b, name)), name
        a.close()
    batch.close()


STAR1, STAR4 = dict(K=32, mini_batch_size=300), dict(K=32, mini_batch_size=3000)
EDGES = dict(K=32, mini_batch_size=400, strategy=3)
SOURCES = dict(K=32, mini_batch_size=400, sampler_max_source=6)
WIDE = dict(K=300, mini_batch_size=1500)


@pytest.mark.parametrize("kinds", [[STAR1, STAR4], [STAR4, STAR1, EDGES], [EDGES, STAR1], [SOURCES, WIDE, STAR4]])
@pytest.mark.parametrize("dtype", [_native.PI_F32, _native.PI_BF16])
def test_commits_of_several_kinds(net, kinds, dtype):
    check(net, [dict(kw, pi_dtype=dtype) for kw in kinds])


def test_update_phi_with_a_launch_per_kind(net, monkeypatch):
    monkeypatch.setenv("AMMSB_PHI_RING", "6")
    check(net, [dict(K=1000, mini_batch_size=m, pi_dtype=_native.PI_F32) for m in (40, 600)])
