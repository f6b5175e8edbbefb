"""A recording of which one step graph finds no memory (SLIME_FAIL_GRAPH, in a
child process): it makes the steps it was asked for, once, and its gradients
are those of an undisturbed recording."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# 65,536 agents and 93 steps: recorded on a sorted copy, in segments of 31 whose
# graphs are one per buffer parity.
CODE = """
import sys
sys.path.insert(0, %r); sys.path.insert(0, %r)
import numpy as np
import slime_gb300 as sg
from conftest import agents_uniform, config0_params
W, H, N, STEPS = 512, 384, 65_536, 93
p = config0_params(W, H, pheromone_deposition_amount=0.01, decay_factor=0.9)
with sg.Simulation(W, H, N, p) as sim:
    sim.upload_agents(agents_uniform(N, W, H, 1.0, 2.0, seed=3))
    sim.upload_trail(np.random.default_rng(4).random((H, W), dtype=np.float32))
    sim.forward_record(STEPS, 31)
    steps = sim.info().steps_done
    g, d_trail = sim.backward(np.random.default_rng(5).standard_normal((H, W)).astype(np.float32))
    np.savez(sys.argv[1], steps=steps, agents=sim.download_agents(), trail=sim.download_trail(), d_trail=d_trail,
             grads=[g.d_decay_factor, g.d_diffusion_rate, g.d_deposition_amount])
""" % (os.path.join(ROOT, "slime-mold_gb300"), os.path.join(ROOT, "tests"))


def record(path, failing):
    env = dict(os.environ, SLIME_FAIL_GRAPH=str(failing))
    out = subprocess.run([sys.executable, "-c", CODE, str(path)], env=env, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    return np.load(path)


def test_a_graph_without_memory_does_not_record_twice(gpu, tmp_path):
    want = record(tmp_path / "want.npz", 0)
    assert want["steps"] == 93
    for failing in (1, 2, 3, 4):
        got = record(tmp_path / f"{failing}.npz", failing)
        assert got["steps"] == 93, f"graph {failing} failing"
        for k in ("agents", "trail", "d_trail", "grads"):
            assert got[k].tobytes() == want[k].tobytes(), f"{k}, graph {failing} failing"
