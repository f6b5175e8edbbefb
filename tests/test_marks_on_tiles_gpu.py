"""Steps that record marks on the shared-memory trail tiles: tiny and odd grids
with at most one agent a cell, and the counts made on demand after the
reference's dispatch, whose agents are visited twice, once or never."""
import numpy as np
import pytest

import oracle
from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", range(1, 8))
@pytest.mark.parametrize("W,H", [(3, 5), (1, 1), (64, 8), (65, 9), (129, 130), (4, 300)])
def test_tiles_fold_marks(gpu, tile, W, H):
    n = max(1, W * H // 2)
    for blur_mode, radius in ((0, 1.0), (1, 0.0), (1, 1.0), (1, 3.0), (1, 8.0)):
        p = config0_params(W, H, decay_mode=blur_mode, decay_factor=0.97 if blur_mode else 10.0, blur_mode=blur_mode,
                           blur_radius=radius, blur_sigma=1.7)
        agents = agents_uniform(n, W, H, 1.0, 2.0, seed=4)
        trail = np.random.default_rng(W + tile).random((H, W), dtype=np.float32)
        with make_sim(W, H, n, p, agents, trail) as sim:
            sim.set_options(trail_tile=tile)
            sim.step(3)
            ca, ct = agents.copy(), trail.copy()
            want = oracle.run(p, W, H, ca, ct, 3, record_counts=True)[-1]
            what = f"{W}x{H} tile {tile} blur {blur_mode} r {radius}"
            assert_bitexact(sim.download_trail(), ct, "trail " + what)
            assert_bitexact(sim.download_agents(), ca, "agents " + what)
            assert_bitexact(sim.download_deposit_counts(), want, "counts " + what)


@pytest.mark.parametrize("reorder", [0, 1])
def test_counts_on_demand_in_the_reference_dispatch(gpu, reorder):
    W, H, n = 2101, 2100, 4_264_240  # more cells than agents
    p = config0_params(W, H, dispatch_mode=1, agent_speed_min=30.0, agent_speed_max=50.0)
    agents = agents_uniform(n, W, H, 30.0, 50.0, seed=8)
    trail = np.random.default_rng(9).random((H, W), dtype=np.float32)
    ca, ct = agents.copy(), trail.copy()
    want = oracle.run(p, W, H, ca, ct, 2, record_counts=True)[-1]
    with make_sim(W, H, n, p, agents, trail) as sim:
        if reorder:
            sim.reorder_agents()
        before = sim.info().kernel_launches
        sim.step(2)
        # marks need no second pass over the agents that are visited twice
        assert sim.info().kernel_launches - before == 2 * 2
        assert_bitexact(sim.download_deposit_counts(), want, "counts")
        assert want.max() > 1 and want.sum() > n  # visited twice
        assert_bitexact(sim.download_trail(), ct, "trail")
        sim.reorder_agents()
        assert_bitexact(sim.download_deposit_counts(), want, "counts after a reorder")
