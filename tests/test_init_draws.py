"""The initial phi draw by draw: the FP32 rounding of the FP64 Gamma(1, 1)
stream, at row lengths with padding and a first element per row anywhere in a
block; the oracle's FP64 draw is within one rounding of it (1.2e-7)."""
import numpy as np
import pytest

import oracle
from mcmc_for_ammsb_gb300 import MCMCSamplerStochastic, Network, Options, _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,dtype", [(2000, 1, _native.PI_F32), (900, 7, _native.PI_BF16),
                                       (333, 33, _native.PI_F32), (40, 300, _native.PI_F32),
                                       (20, 1000, _native.PI_BF16)])
@pytest.mark.parametrize("seed", [1, 2026])
def test_phi_is_the_fp64_stream(native_lib, n, K, dtype, seed):
    net = Network.from_edges(n, np.arange(n - 1), np.arange(1, n))
    net.held_out = net.test = (np.array([0], np.int32), np.array([2], np.int32),
                               np.array([0], np.uint8))
    s = MCMCSamplerStochastic(Options(K=K, num_node_sample=4, mini_batch_size=2, random_seed=seed, chain=3,
                                      pi_dtype=dtype), net).init()
    draw = oracle.lib().oracle_gamma
    want = np.array([[draw(seed, 3, oracle.P_PHI_INIT, v, k, 1.0, 1.0) for k in range(K)] for v in range(n)])
    assert np.all(np.abs(s.phi - want) <= 1.2e-7 * want)
    s.close()
