"""update_phi's ring kernel where its rows and groups have remainders, against
the oracle with the tolerances of test_gpu_parity: chunks of four, two and one
rows (by the floats a lane holds) with 1 to U + 1 rows on a warp, 64 and 65
nodes (16 warps per node, then groups of four), and ring depths of which four
groups do not fit an SM (a launch per kind of iteration, and one group per
CTA)."""
import pytest

from mcmc_for_ammsb_gb300 import Network, _native
from test_gpu_parity import run_fed_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(native_lib):
    net = Network.synthetic(n=1500, k_true=15, intra_degree=6.0, seed=4)
    net.make_held_out(0.02, seed=4)
    return net


@pytest.mark.parametrize("K,dtype", [(256, _native.PI_BF16),   # chunks of 4, whole rows
                                     (250, _native.PI_F32),    # 4, ragged
                                     (300, _native.PI_F32),    # 2
                                     (510, _native.PI_BF16),   # 2, ragged
                                     (1000, _native.PI_F32)])  # 1
@pytest.mark.parametrize("nodes,nns", [(65, 1), (65, 15), (65, 19), (65, 70), (64, 33)])
def test_chunk_and_group_remainders(net, K, dtype, nodes, nns):
    run_fed_case(net, K, 5, dtype, strategy=2, mini_batch_size=nodes - 1, num_node_sample=nns)


@pytest.mark.parametrize("K,dtype", [(1024, _native.PI_BF16), (1000, _native.PI_F32)])
@pytest.mark.parametrize("nodes", [40, 700])
def test_deep_rings_take_a_launch_per_kind(net, monkeypatch, K, dtype, nodes):
    monkeypatch.setenv("AMMSB_PHI_RING", "6")
    run_fed_case(net, K, 5, dtype, strategy=2, mini_batch_size=nodes - 1, num_node_sample=20)


def test_few_nodes_with_groups_of_four(net, monkeypatch):
    monkeypatch.setenv("AMMSB_PHI_FEW", "0")
    run_fed_case(net, 256, 5, _native.PI_BF16, strategy=2, mini_batch_size=9, num_node_sample=20)
