"""Steps run on a sorted copy of the agents when the context does not reorder
them and enough steps are made: the same bits as the oracle's and as a context
that reorders, whatever is done between the steps."""
import numpy as np
import pytest

import oracle
from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,n,steps,speed", [(160, 96, 32768, 64, 40.0), (160, 96, 32767, 64, 40.0),
                                               (203, 131, 40001, 65, 300.0), (512, 64, 200_003, 16, 1.0)])
def test_sorted_run_matches_single_steps_and_the_oracle(gpu, W, H, n, steps, speed):
    p = config0_params(W, H, agent_speed_min=speed / 2, agent_speed_max=speed, agent_jitter=0.2)
    agents = agents_uniform(n, W, H, speed / 2, speed, seed=3)
    trail = np.random.default_rng(4).random((H, W), dtype=np.float32)
    a, b = (make_sim(W, H, n, p, agents, trail) for _ in range(2))
    a.prepare_steps(steps)
    a.step(steps)
    for _ in range(steps):
        b.step(1)
    assert a.info().reordered == 0 and a.info().steps_done == steps
    ca, ct = agents.copy(), trail.copy()
    want = oracle.run(p, W, H, ca, ct, steps, record_counts=True)[-1]
    assert_bitexact(a.download_agents(), ca, "agents")
    assert_bitexact(a.download_trail(), ct, "trail")
    assert_bitexact(a.download_deposit_counts(), want, "counts")
    assert_bitexact(b.download_agents(), ca, "agents, single steps")
    assert_bitexact(b.download_trail(), ct, "trail, single steps")


def test_sorted_runs_between_changes(gpu):
    W, H, n, steps = 160, 96, 40000, 70
    p = config0_params(W, H, agent_speed_min=20.0, agent_speed_max=40.0, agent_jitter=0.2)
    agents = agents_uniform(n, W, H, 20.0, 40.0, seed=3)
    trail = np.random.default_rng(4).random((H, W), dtype=np.float32)
    a, b = (make_sim(W, H, n, p, agents, trail) for _ in range(2))
    b.set_options(reorder_every=7, use_graphs=0)

    def both(what):
        a.step(steps)
        b.step(steps)
        assert_bitexact(a.download_agents(), b.download_agents(), "agents " + what)
        assert_bitexact(a.download_trail(), b.download_trail(), "trail " + what)

    both("first")
    for s in (a, b):
        s.upload_agents(agents)
    both("after an upload")
    a.set_options(use_graphs=0)
    both("without graphs")
    for s in (a, b):
        s.reassign_speeds(5)
    a.set_options(use_graphs=1, exact_counts=1)
    both("counting")
    for s in (a, b):
        s.resize(200, 80)
    both("after a resize")
    for s in (a, b):
        s.set_agent_count(50001, 9)
    both("after another agent count")
    a.reorder_agents()
    both("after a reorder by hand")
    for s in (a, b):
        s.set_params(config0_params(200, 80, agent_speed_min=20.0, agent_speed_max=40.0, dispatch_mode=1))
    both("in the reference's dispatch")


def test_sorted_copy_across_single_steps_and_other_calls(gpu, tmp_path):
    """One step per call, as a display loop makes them: onto the copy after 64
    (of 32,768 agents), and every other entry point while the copy is stepped."""
    W, H, n = 160, 96, 33000
    p = config0_params(W, H, agent_speed_min=20.0, agent_speed_max=40.0, agent_jitter=0.2)
    agents = agents_uniform(n, W, H, 20.0, 40.0, seed=3)
    trail = np.random.default_rng(4).random((H, W), dtype=np.float32)
    lut = np.random.default_rng(5).integers(0, 256, 768).astype(np.uint8)
    a, b = (make_sim(W, H, n, p, agents, trail) for _ in range(2))
    b.set_options(reorder_every=1)

    def both(k, what):
        for _ in range(k):
            a.step(1)
            b.step(1)
        assert_bitexact(a.download_agents(), b.download_agents(), "agents " + what)
        assert_bitexact(a.download_trail(), b.download_trail(), "trail " + what)
        assert np.array_equal(a.colorize(lut, 80, 60), b.colorize(lut, 80, 60)), "image " + what

    both(70, "after 70 frames")
    before = a.info().kernel_launches
    a.step(1)
    assert a.info().kernel_launches - before == 2  # on the copy: no sort for one more step
    b.step(1)
    for s in (a, b):
        s.reassign_speeds(5)
    both(3, "after new speeds")
    a.profile_steps(2)
    b.step(2)
    both(1, "after profiled steps")
    a.save_state(tmp_path / "s")
    c = type(a).load_state(tmp_path / "s")
    both(2, "after a save")
    c.step(2)
    assert_bitexact(c.download_agents(), a.download_agents(), "resumed")
    a.restore_state(tmp_path / "s")
    b.restore_state(tmp_path / "s")
    both(66, "after a restore")
    a.set_steps_done(10)
    both(3, "after another step count")
    g = np.ones((H, W), np.float32)
    grads = []
    for s in (a, b):
        s.forward_record(5, 2)
        r, d0 = s.backward(g)
        grads.append((r.d_decay_factor, r.d_diffusion_rate, r.d_deposition_amount, d0))
    assert_bitexact(grads[0][3], grads[1][3], "dL/dT0")
    both(2, "after a recording")
    a.autotune(1)
    both(70, "after tuning")
    a.set_options(reorder_every=3)
    both(4, "with a schedule")
    a.set_options(reorder_every=0)
    a.reorder_agents()
    both(70, "reordered by hand")
