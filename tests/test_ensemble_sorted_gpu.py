"""An ensemble without a reorder schedule sorts its colonies by itself once
enough steps are made: the same bits as plain runs, in both engines, tuned or
not, single steps or many, and after a colony's agents were set anew."""
import numpy as np
import pytest

from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [None, 0, 1])
@pytest.mark.parametrize("tuned", [False, True])
def test_sorted_by_itself(gpu, engine, tuned):
    import slime_gb300 as sg
    sizes = [(128, 96, 24000), (64, 40, 9000), (8, 8, 0), (132, 20, 1000)]
    params = [config0_params(W, H, agent_speed_min=60.0 + 10 * j, agent_speed_max=120.0, agent_jitter=0.1,
                             pheromone_deposition_amount=1.0 - 0.2 * j) for j, (W, H, _) in enumerate(sizes)]
    ens = sg.Ensemble([s[0] for s in sizes], [s[1] for s in sizes], [s[2] for s in sizes], params)
    assert ens.info().engine == sg.ENSEMBLE_LANES
    if engine is not None:
        ens.set_engine(engine)
    sims = [sg.Simulation(W, H, n, p) for (W, H, n), p in zip(sizes, params)]

    def give(j, seed):
        W, H, n = sizes[j]
        agents = agents_uniform(n, W, H, 60.0, 120.0, seed=seed)
        ens.upload_agents(j, agents)
        sims[j].upload_agents(agents)

    for j, (W, H, n) in enumerate(sizes):
        give(j, j)
        trail = np.random.default_rng(j).random((H, W), dtype=np.float32)
        ens.upload_trail(j, trail)
        sims[j].upload_trail(trail)
    if tuned:
        ens.autotune(1)
        if engine is not None:
            ens.set_engine(engine)

    def both(calls, steps, what):
        for _ in range(calls):
            ens.step(steps)
        ens.sync()
        for j, sim in enumerate(sims):
            for _ in range(calls * steps):
                sim.step(1)
            assert_bitexact(ens.download_agents(j), sim.download_agents(), f"agents of {j} {what}")
            assert_bitexact(ens.download_trail(j), sim.download_trail(), f"trail of {j} {what}")

    ens.prepare_steps(70)
    both(1, 70, "after 70 steps")
    both(20, 1, "after single steps")
    give(0, 50)
    both(3, 1, "after an upload")
    both(1, 64, "after an upload and many steps")
    ens.set_reorder(5, 1)
    both(1, 12, "with a schedule")
    ens.set_reorder(0, 2)
    both(1, 65, "without one again")
