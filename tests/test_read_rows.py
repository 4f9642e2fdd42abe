"""BF16 pi read back: on the host, on the device in one piece and in several with
a ragged last one, with and without padding behind the rows; every value is the
widened one of the checkpoint's raw rows."""
import numpy as np
import pytest

from mcmc_for_ammsb_gb300 import MCMCSamplerStochastic, Network, Options, _native

pytestmark = pytest.mark.gpu


# 16,384 values are the most that the host widens, 2,097,152 a staging buffer's
@pytest.mark.parametrize("n,K", [(10, 3), (2048, 8), (2049, 8), (5000, 7), (262144, 8), (262145, 8), (30001, 250),
                                 (5003, 1024)])
def test_pi_is_the_stored_rows_widened(native_lib, tmp_path, n, K):
    net = Network.from_edges(n, np.arange(n - 1), np.arange(1, n))
    net.held_out = net.test = (np.array([0], np.int32), np.array([2], np.int32), np.array([0], np.uint8))
    s = MCMCSamplerStochastic(Options(K=K, num_node_sample=4, mini_batch_size=2, pi_dtype=_native.PI_BF16), net).init()
    s.save_checkpoint(tmp_path / "chain")
    raw = np.fromfile(tmp_path / "chain", np.uint16)[-n * K:]
    want = (raw.astype(np.uint32) << 16).view(np.float32).reshape(n, K)
    for _ in range(2):
        assert np.array_equal(s.pi, want)
    s.close()
