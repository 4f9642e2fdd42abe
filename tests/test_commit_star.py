"""The commit of a star minibatch (k_commit_star, what ammsb_step launches for
the default strategies) against the commit of a general edge list
(k_commit_beta, what the sharded phases launch): one owner of every node and
edge takes the same iteration, bit for bit."""
import numpy as np
import pytest

from mcmc_for_ammsb_gb300 import MCMCSamplerStochastic, Options, _native, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(native_lib):
    return workloads.build("diff")[0]  # 2,000 nodes


# 1,024 summing warps: one edge each up to 1,024 edges, rounds of four above;
# K around the lanes' four elements and the 128-element pieces of a row
@pytest.mark.parametrize("m", [1, 3, 1024, 1025, 1500])
@pytest.mark.parametrize("K,dtype", [(1, _native.PI_F32), (130, _native.PI_F32),
                                     (7, _native.PI_BF16), (513, _native.PI_BF16)])
def test_star_commit_equals_general_commit(net, m, K, dtype):
    o = dict(K=K, num_node_sample=8, mini_batch_size=m, pi_dtype=dtype)
    a = MCMCSamplerStochastic(Options(**o), net).init()
    b = MCMCSamplerStochastic(Options(**o), net).init()
    flags = set()
    for _ in range(5):
        mb = b.shard_draw()
        rows = b.shard_update(np.arange(len(mb["nodes"])))
        b.shard_theta(b.shard_commit(rows, np.arange(len(mb["edge_a"]))))
        a.step(1)
        flags.add(mb["flag"])
        for name in ("theta", "beta", "pi", "phi"):
            assert np.array_equal(getattr(a, name), getattr(b, name)), name
    assert flags == {0, 1}  # both strata
    a.close()
    b.close()
