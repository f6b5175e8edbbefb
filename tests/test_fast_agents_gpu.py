"""Agents too fast to stay in order step in their slots: a sort pays up to 0.7
cells a step for 32,768 agents, 1 from 100,000, 8 from 200,000, 24 or on large
trails 128 from a million.  Changing the speeds moves them off the copy and back,
with the results of plain steps."""
import numpy as np
import pytest

import oracle
from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


def speeds(cells):
    """Parameters with the fastest agents at `cells` cells a step."""
    return dict(agent_speed_min=cells / 0.016 / 2, agent_speed_max=cells / 0.016)


@pytest.mark.parametrize("W,H,n,steps,slow,fast", [(256, 96, 40_000, 64, 0.69, 0.71), (256, 96, 100_000, 64, 0.99, 1.01),
                                                   (256, 96, 200_000, 16, 7.9, 8.1),
                                                   (1024, 64, 1_000_000, 16, 23.9, 24.1)])
def test_only_agents_that_stay_in_order_are_sorted(gpu, W, H, n, steps, slow, fast):
    for cells, sorts in ((slow, 1), (fast, 0)):
        with make_sim(W, H, n, config0_params(W, H, **speeds(cells)), agents_uniform(n, W, H, 1.0, 500.0, seed=1),
                      np.zeros((H, W), np.float32)) as sim:
            before = sim.info().kernel_launches
            sim.step(steps)
            launches = sim.info().kernel_launches - before
            assert (launches > 2 * steps) == bool(sorts), f"{cells} cells a step: {launches} launches"


def test_speeds_that_change(gpu):
    W, H, n = 256, 96, 200_003
    agents = agents_uniform(n, W, H, 30.0, 900.0, seed=2)
    trail = np.random.default_rng(3).random((H, W), dtype=np.float32)
    a = make_sim(W, H, n, config0_params(W, H, **speeds(1.0)), agents, trail)
    ca, ct = agents.copy(), trail.copy()
    for cells in (1.0, 12.0, 1.0, 0.5):
        p = config0_params(W, H, **speeds(cells))
        a.set_params(p)
        a.step(20)
        oracle.run(p, W, H, ca, ct, 20)
        assert_bitexact(a.download_agents(), ca, f"agents at {cells} cells a step")
        assert_bitexact(a.download_trail(), ct, f"trail at {cells} cells a step")


def test_ensembles_sort_only_their_slow_colonies(gpu):
    import slime_gb300 as sg
    W, H, n = 128, 96, 210_000
    p = [config0_params(W, H, **speeds(c)) for c in (2.0, 12.0)]
    ens = sg.Ensemble([W, W], [H, H], [n, n], p)
    sims = [sg.Simulation(W, H, n, q) for q in p]
    for j, sim in enumerate(sims):
        agents = agents_uniform(n, W, H, 60.0, 900.0, seed=j)
        ens.upload_agents(j, agents)
        sim.upload_agents(agents)
    ens.set_engine(sg.ENSEMBLE_LANES)
    before = ens.launch_count()
    ens.step(40)
    assert ens.launch_count() - before == 40 * 2 * 2 + 6 * 3  # the slow one's sorts, every 16 steps
    for j, sim in enumerate(sims):
        sim.step(40)
        assert_bitexact(ens.download_agents(j), sim.download_agents(), f"agents of {j}")
        assert_bitexact(ens.download_trail(j), sim.download_trail(), f"trail of {j}")
