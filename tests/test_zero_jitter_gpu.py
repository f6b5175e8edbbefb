"""Without jitter the hash is not worked out: the headings must still come out as
if it were added times zero, also for a heading of -0 (whose sign the zero
decides) and for positions whose hash is not a number, for every agent shape;
and a jitter of -0 is one of 0."""
import numpy as np
import pytest

import oracle
from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jitter", [0.0, -0.0])
@pytest.mark.parametrize("shape", range(17))
def test_zero_jitter(gpu, shape, jitter):
    W, H = 64, 48
    agents = agents_uniform(1003, W, H, 1.0, 60.0, seed=5)
    agents[:300, 2] = -0.0
    agents[300:330, 2] = 0.0
    agents[330:340, 0] = 1e37  # finite position, infinite hash argument
    agents[340:350, 1] = -3e38
    agents[350:353, 0] = (np.nan, np.inf, -np.inf)
    agents[353:360, 0] = 1e31  # the hash is finite, the position far from the grid
    agents[360:370, 3] = 0.0
    trail = np.random.default_rng(6).random((H, W), dtype=np.float32)
    trail[: H // 2] = 0.0  # no turn there: the heading is the jittered one
    p = config0_params(W, H, agent_jitter=jitter, agent_speed_min=0.0, agent_speed_max=100.0)
    sim = make_sim(W, H, len(agents), p, agents, trail)
    sim.set_options(agent_shape=shape)
    ca, ct = agents.copy(), trail.copy()
    sim.step(3)
    oracle.run(p, W, H, ca, ct, 3)
    assert_bitexact(sim.download_agents(), ca, "agents")
    assert_bitexact(sim.download_trail(), ct, "trail")
