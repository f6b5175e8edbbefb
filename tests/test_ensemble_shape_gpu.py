"""Which engine steps an ensemble that was neither tuned nor told: the
cooperative one where a launch shape of it was chosen by hand, where many small
colonies make few steps at a time, and just after parameters were set."""
import numpy as np
import pytest

from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact

pytestmark = pytest.mark.gpu


def test_a_shape_by_hand_steps_cooperatively(gpu):
    import slime_gb300 as sg

    def ensemble():
        return sg.Ensemble([64, 128], [32, 64], [500, 3000], [config0_params(64, 32), config0_params(128, 64)])

    ens = ensemble()
    ens.set_shape(16, 2, 2)
    assert ens.info().engine == sg.ENSEMBLE_COOPERATIVE
    before = ens.launch_count()
    ens.step(7)
    assert ens.launch_count() - before == 7  # one launch a step
    ens = ensemble()
    ens.set_engine(sg.ENSEMBLE_LANES)
    ens.set_shape(16, 2, 2)
    assert ens.info().engine == sg.ENSEMBLE_LANES
    ens = ensemble()
    ens.autotune(1)
    tuned = ens.info().engine
    ens.set_shape(16, 2, 2)
    assert ens.info().engine == tuned


def test_the_untuned_engine_follows_the_calls(gpu):
    import slime_gb300 as sg
    k, W, H, n = 12, 64, 40, 1500
    params = [config0_params(W, H, agent_speed_min=20.0, agent_speed_max=40.0, diffusion_rate=0.1 + 0.05 * j,
                             pheromone_deposition_amount=1.0 if j % 3 else 0.4) for j in range(k)]
    ens = sg.Ensemble([W] * k, [H] * k, [n] * k, params)
    sims = [sg.Simulation(W, H, n, p) for p in params]
    for j, sim in enumerate(sims):
        agents = agents_uniform(n, W, H, 20.0, 40.0, seed=j)
        ens.upload_agents(j, agents)
        sim.upload_agents(agents)

    def step(m, engine, what):
        before = ens.launch_count()
        ens.step(m)
        assert ens.info().engine == engine, what
        assert ens.launch_count() - before == (m if engine == sg.ENSEMBLE_COOPERATIVE else 2 * k * m), what
        for sim in sims:
            sim.step(m)

    def compare(what):
        for j, sim in enumerate(sims):
            assert_bitexact(ens.download_agents(j), sim.download_agents(), f"agents of {j} {what}")
            assert_bitexact(ens.download_trail(j), sim.download_trail(), f"trail of {j} {what}")

    coop, lanes = sg.ENSEMBLE_COOPERATIVE, sg.ENSEMBLE_LANES
    step(7, lanes, "with the parameters of the creation")
    step(2, coop, "two steps of twelve colonies")
    compare("after both engines")
    for r in range(3):
        step(1, coop, "single steps between")
        step(7, lanes, "longer calls")
    compare("after alternating calls")
    for j in (0, 5):
        params[j].decay_factor = 0.9
        params[j].pheromone_deposition_amount = 1.4 - params[j].pheromone_deposition_amount  # marks on and off
        ens.set_params(j, params[j])
        sims[j].set_params(params[j])
    step(7, coop, "after new parameters")
    step(7, lanes, "and again")
    compare("after new parameters")
    ens.set_params(0, params[0])
    ens.prepare_steps(14)
    step(14, lanes, "prepared")
    compare("after a prepared call")
