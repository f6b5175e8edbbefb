"""Deposits added up within a warp, on both sides of four agents a cell: agents
all over the grid, most of them in a few cells, and all in one, with a last
group that is not full; counts, trail and agents are the oracle's."""
import numpy as np
import pytest

import oracle
from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [10, 12, 14, 15, 16])  # the persistent kernels
@pytest.mark.parametrize("n", [4 * 64 * 48 - 1, 4 * 64 * 48, 40_003])
@pytest.mark.parametrize("spread", ["all", "few", "one"])
def test_crowded_deposits(gpu, shape, n, spread):
    W, H = 64, 48
    agents = agents_uniform(n, W, H, 0.0, 1.0, seed=n)
    if spread == "few":  # five agents in six within a patch of 3 x 2 cells
        agents[n // 6:, 0] = 10.0 + agents[n // 6:, 0] * (3.0 / W)
        agents[n // 6:, 1] = 20.0 + agents[n // 6:, 1] * (2.0 / H)
    elif spread == "one":
        agents[:, 0], agents[:, 1] = 30.5, 30.5
    trail = np.random.default_rng(6).random((H, W), dtype=np.float32)
    p = config0_params(W, H, pheromone_deposition_amount=1e-3, agent_speed_min=0.0, agent_speed_max=1.0)
    sim = make_sim(W, H, n, p, agents, trail)
    sim.set_options(agent_shape=shape, reorder_every=1)
    ca, ct = agents.copy(), trail.copy()
    sim.step(2)
    oracle.run(p, W, H, ca, ct, 2)
    assert_bitexact(sim.download_agents(), ca, "agents")
    assert_bitexact(sim.download_trail(), ct, "trail")
    cells = ca[:, 1].astype(np.int64) * W + ca[:, 0].astype(np.int64)
    assert np.array_equal(sim.download_deposit_counts().reshape(-1), np.bincount(cells, minlength=W * H))
