"""A context without a schedule is tuned on the sorted copy of its agents that
its steps will run on, and left with its state as it was."""
import numpy as np
import pytest

from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,before", [(200_003, 0), (200_003, 20), (40_000, 70), (20_000, 5)])
def test_tuned_in_the_order_of_the_steps(gpu, n, before):
    W, H = 256, 96
    p = config0_params(W, H, agent_speed_min=5.0, agent_speed_max=10.0)
    agents = agents_uniform(n, W, H, 5.0, 10.0, seed=1)
    trail = np.random.default_rng(2).random((H, W), dtype=np.float32)
    a, b = (make_sim(W, H, n, p, agents, trail) for _ in range(2))
    for sim in (a, b):
        if before:
            sim.step(before)
    a.autotune(1)
    assert_bitexact(a.download_agents(), b.download_agents(), "agents after tuning")
    assert_bitexact(a.download_trail(), b.download_trail(), "trail after tuning")
    launches = a.info().kernel_launches
    a.step(16)
    assert a.info().kernel_launches - launches == 2 * 16  # sorted already, or too few to be
    for _ in range(16):
        b.step(1)
    assert_bitexact(a.download_agents(), b.download_agents(), "agents")
    assert_bitexact(a.download_trail(), b.download_trail(), "trail")
