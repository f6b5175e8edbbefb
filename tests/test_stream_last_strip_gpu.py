"""Streaming trail strips whose last one is a single 4-column group (widths of
128 k + 4): that lane is the strip's first and last, and needs the halo cells
of both its sides."""
import numpy as np
import pytest

import oracle
from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [8, 9, 10])
@pytest.mark.parametrize("W,H", [(132, 40), (260, 9), (128, 9)])
def test_last_strip_of_one_lane(gpu, tile, W, H):
    n = 2000
    for blur_mode, radius, exact_counts in ((0, 1.0, 1), (1, 1.0, 0), (1, 2.0, 1)):
        p = config0_params(W, H, blur_mode=blur_mode, blur_radius=radius, blur_sigma=1.3)
        agents = agents_uniform(n, W, H, 1.0, 2.0, seed=4)
        trail = np.random.default_rng(5).random((H, W), dtype=np.float32)
        sim = make_sim(W, H, n, p, agents, trail)
        sim.set_options(trail_tile=tile, exact_counts=exact_counts)
        sim.step(2)
        ca, ct = agents.copy(), trail.copy()
        oracle.run(p, W, H, ca, ct, 2)
        assert_bitexact(sim.download_trail(), ct, f"trail {W}x{H} tile {tile} blur {blur_mode} r {radius}")
        sim.close()


def test_ensemble_colony_of_that_width(gpu):
    import slime_gb300 as sg
    W, H, n = 132, 64, 2000
    p = config0_params(W, H)
    agents = agents_uniform(n, W, H, 1.0, 2.0, seed=6)
    trail = np.random.default_rng(7).random((H, W), dtype=np.float32)
    ca, ct = agents.copy(), trail.copy()
    oracle.run(p, W, H, ca, ct, 2)
    for engine in (sg.ENSEMBLE_COOPERATIVE, sg.ENSEMBLE_LANES):
        ens = sg.Ensemble([W, 128], [H, 32], [n, 100], [p, config0_params(128, 32)])
        ens.set_engine(engine)
        ens.upload_agents(0, agents)
        ens.upload_trail(0, trail)
        ens.step(2)
        assert_bitexact(ens.download_trail(0), ct, "colony trail")
        ens.close()
