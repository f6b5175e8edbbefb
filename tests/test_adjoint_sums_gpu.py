"""The backward's parameter sums are held in binary64 over cells and steps: in
range and in precision beyond what binary32 numbers, single or in pairs, hold."""
import numpy as np
import pytest

from conftest import config0_params
from test_parity_gpu import make_sim

pytestmark = pytest.mark.gpu

W, H = 140, 40


def decay_gradient(g, steps):
    """A trail of 0.5 that neither decays nor spreads: d_decay_factor is half the
    sum of g, once per step, with every product exact."""
    p = config0_params(W, H, pheromone_deposition_amount=0.1, decay_factor=1.0, diffusion_rate=0.0)
    with make_sim(W, H, 0, p, np.zeros((0, 4), np.float32), np.full((H, W), 0.5, np.float32)) as sim:
        sim.forward_record(steps, 3)
        return sim.backward(g)[0].d_decay_factor


def test_sums_over_steps_beyond_the_binary32_range(gpu):
    g = np.full((H, W), 1e38, np.float32)  # four cells of a column: 2e38, twice that is no binary32
    for steps in (1, 2, 8):
        got, want = decay_gradient(g, steps), 0.5 * steps * W * H * float(np.float32(1e38))
        assert np.isfinite(got) and abs(got - want) <= 1e-12 * want, f"{steps} steps"


@pytest.mark.parametrize("steps", [1, 4])
def test_sums_of_53_bits(gpu, steps):
    # neighbouring columns: 2^50 and down to 1, exact in binary64 and in nothing shorter
    g = np.zeros((H, W), np.float32)
    g[0, 0], g[0, 1], g[0, 2] = (2.0**24 - 1) * 2.0**26, (2.0**24 - 1) * 2.0**3, 1.0
    exact = [int(v) for v in g[0, :3]]
    assert all(float(e) == v for e, v in zip(exact, g[0, :3]))
    assert decay_gradient(g, steps) == 0.5 * steps * sum(exact)
