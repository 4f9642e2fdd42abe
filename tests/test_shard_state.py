"""A sharded iteration's theta step after the state was set anew: it starts from
the theta of now, not from the one that the commit saw."""
import numpy as np
import pytest

from mcmc_for_ammsb_gb300 import MCMCSamplerStochastic, Options, workloads

pytestmark = pytest.mark.gpu


# set_state clears the drawn iteration's step size and scale, so the step that
# follows moves nothing: exact
@pytest.mark.parametrize("K", [7, 40])
def test_theta_step_follows_a_set_state(native_lib, K):
    net = workloads.build("diff")[0]
    s = MCMCSamplerStochastic(Options(K=K, num_node_sample=8, mini_batch_size=50), net).init()
    mb = s.shard_draw()
    R = s.shard_commit(s.shard_update(np.arange(len(mb["nodes"]))), np.arange(len(mb["edge_a"])))
    rng = np.random.default_rng(K)
    theta = rng.gamma(1.0, 1.0, (K, 2)) + 0.1
    s.set_state(s.phi, theta)
    s.shard_theta(R)
    assert np.array_equal(s.theta, theta)
    assert np.array_equal(s.beta, (theta[:, 1] / (theta[:, 0] + theta[:, 1])).astype(np.float32))
