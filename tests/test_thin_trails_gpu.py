"""Trails much longer than wide: their agents are sorted with a key of as many
bits as the sides need, in little memory (the library's allocations are capped
in a child process), with the results of unsorted steps."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, agents_uniform, config0_params
from test_parity_gpu import assert_bitexact

pytestmark = pytest.mark.gpu

HEAD = """
import sys
sys.path.insert(0, %r); sys.path.insert(0, %r)
import numpy as np
import slime_gb300 as sg
from conftest import agents_uniform, config0_params
""" % (os.path.join(ROOT, "slime-mold_gb300"), os.path.join(ROOT, "tests"))


def child(code, cap):
    env = dict(os.environ, SLIME_DEVICE_MEMORY_CAP=str(cap))
    out = subprocess.run([sys.executable, "-c", HEAD + code], env=env, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr


def params(W, H):
    return config0_params(W, H, agent_speed_min=60.0, agent_speed_max=125.0)


# A square code for these sides would take a histogram of 1 to 16 GiB.
@pytest.mark.parametrize("W,H", [(131_076, 8), (8, 131_080), (65_536, 16), (100_003, 5), (3, 262_144)])
def test_sorted_steps_and_reorders(gpu, tmp_path, W, H):
    import slime_gb300 as sg
    n, steps = 200_000, 40
    code = f"""
W, H, n = {W}, {H}, {n}
out = {{}}
for by_hand in (0, 1):
    with sg.Simulation(W, H, n, config0_params(W, H, agent_speed_min=60.0, agent_speed_max=125.0)) as sim:
        sim.upload_agents(agents_uniform(n, W, H, 60.0, 125.0, seed=1))
        before = sim.info().kernel_launches
        if by_hand:
            sim.reorder_agents()
        sim.step({steps})
        out[f"launches{{by_hand}}"] = sim.info().kernel_launches - before
        out[f"a{{by_hand}}"], out[f"t{{by_hand}}"] = sim.download_agents(), sim.download_trail()
np.savez({str(tmp_path / "out.npz")!r}, **out)
"""
    child(code, 96 << 20)
    got = np.load(tmp_path / "out.npz")
    # two kernels a step, six a sort: at the start and every 16 steps, or by hand
    assert got["launches0"] == 2 * steps + 6 * 3
    assert got["launches1"] == 2 * steps + 6
    with sg.Simulation(W, H, n, params(W, H)) as sim:
        sim.upload_agents(agents_uniform(n, W, H, 60.0, 125.0, seed=1))
        for _ in range(5):  # eight steps at a time, too few to be sorted for
            sim.step(8)
            sim.upload_agents(sim.download_agents())
        want = sim.download_agents(), sim.download_trail()
    for by_hand in (0, 1):
        assert_bitexact(got[f"a{by_hand}"], want[0], f"agents, by_hand {by_hand}")
        assert_bitexact(got[f"t{by_hand}"], want[1], f"trail, by_hand {by_hand}")


def test_ensemble_of_thin_colonies(gpu, tmp_path):
    import slime_gb300 as sg
    sizes = [(65_536, 16, 120_000), (131_076, 8, 100_000)]
    code = f"""
sizes = {sizes}
ens = sg.Ensemble([s[0] for s in sizes], [s[1] for s in sizes], [s[2] for s in sizes],
                  [config0_params(W, H, agent_speed_min=60.0, agent_speed_max=125.0) for W, H, n in sizes])
for j, (W, H, n) in enumerate(sizes):
    ens.upload_agents(j, agents_uniform(n, W, H, 60.0, 125.0, seed=j))
ens.set_engine(sg.ENSEMBLE_LANES)
before = ens.launch_count()
ens.step(70)
np.savez({str(tmp_path / "out.npz")!r}, launches=ens.launch_count() - before,
         **{{f"a{{j}}": ens.download_agents(j) for j in range(2)}}, **{{f"t{{j}}": ens.download_trail(j) for j in range(2)}})
"""
    child(code, 96 << 20)
    got = np.load(tmp_path / "out.npz")
    assert got["launches"] == 70 * 2 * 2 + 5 * 2 * 6
    for j, (W, H, n) in enumerate(sizes):
        with sg.Simulation(W, H, n, params(W, H)) as sim:
            sim.upload_agents(agents_uniform(n, W, H, 60.0, 125.0, seed=j))
            sim.step(70)
            assert_bitexact(got[f"a{j}"], sim.download_agents(), f"agents of {j}")
            assert_bitexact(got[f"t{j}"], sim.download_trail(), f"trail of {j}")
