"""The sorted copy and its scratch make room for a resize and for another agent
count, which fit without them (the library's allocations are capped in a child
process)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# 200,000 agents take 3.2 MB, their upload's buffer as much, the copy 4 and its
# sort's scratch 4.8; the trails of 256 x 96 cells 0.5.
CODE = """
import sys
sys.path.insert(0, %r); sys.path.insert(0, %r)
import numpy as np
import slime_gb300 as sg
from conftest import agents_uniform, config0_params
W, H, n = 256, 96, 200_000
with sg.Simulation(W, H, n, config0_params(W, H)) as sim:
    sim.upload_agents(agents_uniform(n, W, H, 1.0, 2.0))
    before = sim.info().kernel_launches
    sim.step(20)
    assert sim.info().kernel_launches - before == 2 * 20 + 6  # on the copy
    {call}
    sim.step(2)
""" % (os.path.join(ROOT, "slime-mold_gb300"), os.path.join(ROOT, "tests"))


# trails of 688^2 cells are 8.6 MB; 500,000 agents 8
@pytest.mark.parametrize("call,cap", [("sim.resize(688, 688)", 17), ("sim.set_agent_count(500_000)", 16)])
def test_room_for_other_sizes(gpu, call, cap):
    env = dict(os.environ, SLIME_DEVICE_MEMORY_CAP=str(cap * 10**6))
    out = subprocess.run([sys.executable, "-c", CODE.replace("{call}", call)], env=env, capture_output=True, text=True,
                         timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
