"""Steps that sort by themselves replay graphs of few lengths: calls of the same
number of steps capture no new ones as the sorted order ages, and a display
loop's single steps none but their own.  SLIME_FAIL_GRAPH makes the first graph
too many fail, in a child process."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HEAD = """
import sys
sys.path.insert(0, %r); sys.path.insert(0, %r)
import slime_gb300 as sg
from conftest import agents_uniform, config0_params
W, H, n = 256, 192, 200_003
p = config0_params(W, H, agent_speed_min=20.0, agent_speed_max=43.75)  # 0.7 cells a step: sorted every 45 steps
agents = agents_uniform(n, W, H, 20.0, 43.75, seed=1)
""" % (os.path.join(ROOT, "slime-mold_gb300"), os.path.join(ROOT, "tests"))


def child(code, graphs):
    env = dict(os.environ, SLIME_FAIL_GRAPH=str(graphs + 1))
    out = subprocess.run([sys.executable, "-c", HEAD + code], env=env, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr


# calls of 100: chunks of 45, 45 and 10 from either buffer; single steps: 15 in
# slot order and the rest on the copy, from either buffer
@pytest.mark.parametrize("calls,steps,graphs", [(25, 100, 4), (300, 1, 4), (40, 7, 4)])
def test_contexts(gpu, calls, steps, graphs):
    child(f"""
with sg.Simulation(W, H, n, p) as sim:
    sim.upload_agents(agents)
    for _ in range({calls}):
        sim.step({steps})
    assert sim.info().steps_done == {calls * steps}
""", graphs)


@pytest.mark.parametrize("calls,steps,graphs", [(25, 100, 4), (40, 7, 2)])
def test_ensembles(gpu, calls, steps, graphs):
    child(f"""
ens = sg.Ensemble([W], [H], [n], [p])
ens.upload_agents(0, agents)
ens.set_engine(sg.ENSEMBLE_LANES)
for _ in range({calls}):
    ens.step({steps})
    assert ens.info().graphs_in_use == 1
assert ens.info().steps_done == {calls * steps}
""", graphs)
