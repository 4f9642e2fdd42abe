"""The initial phi is the FP32 rounding of the FP64 Gamma(1, 1) stream, in enough
draws that several hundred are undecided by the pairs of FP32 numbers and made in
FP64.  The host's FP64 library functions may round other than the device's,
which moves a draw across a rounding boundary about once in 1e8: one draw of the
1.5 million may differ."""
import numpy as np
import pytest

import oracle
from mcmc_for_ammsb_gb300 import MCMCSamplerStochastic, Network, Options

pytestmark = pytest.mark.gpu


def test_every_draw_is_the_rounded_fp64_draw(native_lib):
    n, K = 6000, 250
    net = Network.from_edges(n, np.arange(n - 1), np.arange(1, n))
    net.held_out = net.test = (np.array([0], np.int32), np.array([2], np.int32), np.array([0], np.uint8))
    s = MCMCSamplerStochastic(Options(K=K, num_node_sample=4, mini_batch_size=2, random_seed=11, chain=5), net).init()
    draw = oracle.lib().oracle_gamma
    want = np.array([[draw(11, 5, oracle.P_PHI_INIT, v, k, 1.0, 1.0) for k in range(K)] for v in range(n)])
    assert np.count_nonzero(s.phi != want.astype(np.float32)) <= 1
