"""update_phi's register kernel where its chunks of rows, sub-groups and node
slots have remainders, against the oracle with the tolerances of
test_gpu_parity: chunks of four, two and one rows, sub-groups with no row to
one past a chunk, the last CTA with one node and with all."""
import pytest

from mcmc_for_ammsb_gb300 import Network, _native
from test_gpu_parity import run_fed_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(native_lib):
    net = Network.synthetic(n=900, k_true=9, intra_degree=5.0, seed=6)
    net.make_held_out(0.02, seed=6)
    return net


@pytest.mark.parametrize("K,dtype", [(3, _native.PI_F32), (16, _native.PI_F32), (50, _native.PI_F32),
                                     (8, _native.PI_BF16), (100, _native.PI_BF16)])
@pytest.mark.parametrize("nns,m", [(1, 15), (7, 1), (31, 16), (35, 33), (130, 64)])
def test_narrow_rows(net, K, dtype, nns, m):
    run_fed_case(net, K, 5, dtype, strategy=2, mini_batch_size=m, num_node_sample=nns)


@pytest.mark.parametrize("K,dtype", [(256, _native.PI_F32), (300, _native.PI_F32), (500, _native.PI_BF16)])
@pytest.mark.parametrize("nns", [2, 19])
def test_wide_rows_on_the_register_kernel(net, monkeypatch, K, dtype, nns):
    monkeypatch.setenv("AMMSB_PHI_KERNEL", "regs")
    run_fed_case(net, K, 5, dtype, strategy=2, mini_batch_size=9, num_node_sample=nns)
