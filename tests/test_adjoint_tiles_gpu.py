"""The backward step at the sizes where its tiles can go wrong (widths that are
not whole 16-byte groups, grids smaller than a tile or than the blur, every kind
of blur), against the binary64 adjoint of the same chain; a second recording in
the first one's buffers; sums beyond the binary32 range; a recording long enough
to run on a sorted copy of the agents."""
import numpy as np
import pytest

from conftest import agents_uniform, config0_params
from test_adjoint_gpu import assert_rel, run_case
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,n", [(131, 37, 900), (260, 33, 1500), (7, 5, 20), (128, 16, 400), (129, 17, 400)])
@pytest.mark.parametrize("bm,radius", [(0, 1.0), (1, 0.0), (1, 1.0), (1, 3.0), (1, 5.0), (1, 8.0)])
def test_backward_tiles(gpu, W, H, n, bm, radius):
    steps = 9
    p, t0, counts, theta, grads, d0, ref, d0_ref, g = run_case(W, H, n, steps, 4, 1, bm, 0.05, seed=W, radius=radius,
                                                               t_lo=0.05, decay=0.9)
    got = [grads.d_decay_factor, grads.d_diffusion_rate, grads.d_deposition_amount]
    # every step rounds each term (2 (2R + 1) taps, mixes and products) once per
    # operation: the sum of that many half ulps bounds the relative error
    tol = steps * (4 * radius + 20) * 2.0 ** -24
    for i in range(3):
        if radius == 0.0 and bm == 1 and i == 1:
            assert abs(got[1]) <= 1e-6 * np.abs(g).sum()  # B(u) = u: the rate has no effect
            continue
        assert_rel(got[i], ref[i], f"parameter {i}", tol=tol)
    assert np.max(np.abs(d0 - d0_ref)) <= tol * np.max(np.abs(d0_ref))


def test_a_second_recording_in_the_same_buffers(gpu):
    """200,003 agents and 20 steps: on a sorted copy.  The same recording again,
    one of other parameters, and one of another length, each as on a fresh
    context."""
    W, H, n = 256, 96, 200_003
    agents = agents_uniform(n, W, H, 30.0, 50.0, seed=1)
    trail = (np.random.default_rng(2).random((H, W)) * 0.3 + 0.05).astype(np.float32)
    g = np.random.default_rng(3).random((H, W)).astype(np.float32)

    def record(sim, p, steps):
        sim.set_params(p)
        sim.upload_agents(agents)
        sim.upload_trail(trail)
        sim.forward_record(steps, 8)
        out, a = sim.download_trail(), sim.download_agents()
        grads, d0 = sim.backward(g)
        return out, a, np.array([grads.d_decay_factor, grads.d_diffusion_rate, grads.d_deposition_amount]), d0

    p0 = config0_params(W, H, pheromone_deposition_amount=1e-3, decay_factor=0.9, agent_speed_min=30.0,
                        agent_speed_max=50.0)
    p1 = config0_params(W, H, pheromone_deposition_amount=2e-3, decay_factor=0.8, agent_speed_min=30.0,
                        agent_speed_max=50.0, diffusion_rate=0.3)
    one = make_sim(W, H, n, p0, agents, trail)
    for p, steps in ((p0, 20), (p0, 20), (p1, 20), (p1, 17), (p0, 5)):
        got = record(one, p, steps)
        want = record(make_sim(W, H, n, p, agents, trail), p, steps)
        for x, y, what in zip(got, want, ("trail", "agents", "gradients", "dL/dT0")):
            assert_bitexact(x.astype(np.float32), y.astype(np.float32), f"{what}, {steps} steps")
        plain = make_sim(W, H, n, p, agents, trail)
        for _ in range(steps):
            plain.step(1)
        assert_bitexact(got[0], plain.download_trail(), "trail against plain steps")
        assert_bitexact(got[1], plain.download_agents(), "agents against plain steps")


def test_sums_beyond_binary32_and_special_values(gpu):
    W, H = 140, 40
    p = config0_params(W, H, pheromone_deposition_amount=0.1, decay_factor=1.0, diffusion_rate=0.0)
    trail = np.full((H, W), 0.5, np.float32)
    sim = make_sim(W, H, 0, p, np.zeros((0, 4), np.float32), trail)
    sim.forward_record(1, 1)
    grads, d0 = sim.backward(np.full((H, W), 1e36, np.float32))
    assert np.isfinite(grads.d_decay_factor)  # 5600 terms of 5e35: above the binary32 range
    assert_rel(grads.d_decay_factor, 0.5 * W * H * float(np.float32(1e36)), "sum", tol=1e-6)
    g = np.ones((H, W), np.float32)
    g[3, 5] = np.inf
    # the blur's share of an infinite g at rate 0 is 0 * inf: NaN, in any precision
    assert np.isnan(sim.backward(g)[0].d_decay_factor)
    g[3, 5] = np.nan
    assert np.isnan(sim.backward(g)[0].d_decay_factor)
