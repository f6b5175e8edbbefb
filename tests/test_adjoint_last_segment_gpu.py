"""The last segment of a recording keeps its trails and counts for the backward:
what the recording leaves behind is what the same plain steps leave, a backward
from the kept segment is bit for bit the one that replays every segment, and the
steps after it go on as they would."""
import numpy as np
import pytest

from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


def backward(sim, g):
    grads, d0 = sim.backward(g)
    return np.array([grads.d_decay_factor, grads.d_diffusion_rate, grads.d_deposition_amount]).view(np.uint64), d0


@pytest.mark.parametrize("graphs", [1, 0])
@pytest.mark.parametrize("deposition", [1.0, 1e-3])
@pytest.mark.parametrize("W,H,n,steps,every", [(96, 64, 3000, 20, 8), (96, 64, 3000, 16, 8), (131, 37, 900, 5, 8),
                                               (131, 37, 900, 1, 1), (64, 48, 9000, 7, 1),
                                               (256, 96, 200_003, 37, 17)])
def test_recording_keeps_its_last_segment(gpu, W, H, n, steps, every, deposition, graphs):
    p = config0_params(W, H, pheromone_deposition_amount=deposition, decay_factor=0.9)
    agents = agents_uniform(n, W, H, 1.0, 2.0, seed=1)
    trail = (np.random.default_rng(2).random((H, W)) * 0.3 + 0.05).astype(np.float32)
    g = np.random.default_rng(3).random((H, W)).astype(np.float32)
    sim, plain = make_sim(W, H, n, p, agents, trail), make_sim(W, H, n, p, agents, trail)
    sim.set_options(use_graphs=graphs)
    for again in range(2):  # the second recording: in the first one's buffers, from the other parity where steps is odd
        sim.forward_record(steps, every)
        for _ in range(steps):
            plain.step(1)
        assert_bitexact(sim.download_trail(), plain.download_trail(), "trail")
        assert_bitexact(sim.download_agents(), plain.download_agents(), "agents")
        assert np.array_equal(sim.download_deposit_counts(), plain.download_deposit_counts())
        first, second = backward(sim, g), backward(sim, g)  # the second replays where there are two segments
        assert np.array_equal(first[0], second[0])
        assert_bitexact(first[1], second[1], "dL/dT0")
        sim.step(3 - again)
        plain.step(3 - again)
        assert_bitexact(sim.download_trail(), plain.download_trail(), "trail of later steps")
        third = backward(sim, g)
        assert np.array_equal(first[0], third[0])
        assert_bitexact(first[1], third[1], "dL/dT0 after later steps")
