"""Ensembles that sort their colonies by themselves, where memory or a
colony's shape stands in the way: the steps go on and their results are those
of plain runs.  The library's allocations are capped in a child process
(SLIME_DEVICE_MEMORY_CAP)."""
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


def capped(code, cap, timeout=120):
    """Runs `code` with the library's allocations capped at `cap` bytes."""
    env = dict(os.environ, SLIME_DEVICE_MEMORY_CAP=str(cap))
    out = subprocess.run([sys.executable, "-c", HEAD + code], env=env, capture_output=True, text=True, timeout=timeout)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout


K, SIDE, N = 4, 64, 60_000  # colonies sorted every 16 steps: their fastest agents cross 2 cells a step


def params(j):
    return config0_params(SIDE, SIDE, agent_speed_min=60.0 + j, agent_speed_max=125.0, agent_jitter=0.1)


# A sort takes 24 N bytes and a little; four lanes want that four times.
# Agents, ids and the upload's buffer are 96 N, autotune's snapshot 64 N; 40
# bytes a cell cover the trails, the counts and their snapshot.
@pytest.mark.parametrize("cap_n,tune", [(150, False), (188, True)])
def test_steps_go_on_when_a_later_sort_finds_no_memory(gpu, tmp_path, cap_n, tune):
    import slime_gb300 as sg
    path = tmp_path / "out.npz"
    code = f"""
K, S, N = {K}, {SIDE}, {N}
ens = sg.Ensemble([S] * K, [S] * K, [N] * K,
                  [config0_params(S, S, agent_speed_min=60.0 + j, agent_speed_max=125.0, agent_jitter=0.1) for j in range(K)])
ens.set_engine(sg.ENSEMBLE_COOPERATIVE)
for j in range(K):
    ens.upload_agents(j, agents_uniform(N, S, S, 60.0, 125.0, seed=j))
ens.step(70)
ens.set_engine(sg.ENSEMBLE_LANES)
ens.step(1)
if {tune}:
    ens.autotune(1)
before = ens.launch_count()
ens.step(40)
ens.step(9)
launches = ens.launch_count() - before
np.savez({str(path)!r}, **{{f"a{{j}}": ens.download_agents(j) for j in range(K)}},
         **{{f"t{{j}}": ens.download_trail(j) for j in range(K)}}, steps=ens.info().steps_done, launches=launches)
"""
    capped(code, cap_n * N + 40 * K * SIDE * SIDE)
    got = np.load(path)
    assert got["steps"] == 120
    # two kernels a step and colony at most; three sorts would take 18 more each
    assert got["launches"] <= 49 * K * 2 + 6 * (K - 1)
    for j in range(K):
        with sg.Simulation(SIDE, SIDE, N, params(j)) as sim:
            sim.upload_agents(agents_uniform(N, SIDE, SIDE, 60.0, 125.0, seed=j))
            sim.step(120)
            assert_bitexact(got[f"a{j}"], sim.download_agents(), f"agents of {j}")
            assert_bitexact(got[f"t{j}"], sim.download_trail(), f"trail of {j}")


@pytest.mark.parametrize("engine", [0, 1])
@pytest.mark.parametrize("tuned", [False, True])
def test_colonies_too_wide_to_sort_step(gpu, engine, tuned):
    """A side of more than 262,144 cells has no sort key: such a colony steps as
    its agents come, the others of the ensemble are sorted.  By a schedule it
    is still refused."""
    import slime_gb300 as sg
    sizes = [(262_148, 8, 150_000), (128, 96, 210_000)]
    params = [config0_params(W, H, agent_speed_min=60.0, agent_speed_max=125.0) for W, H, _ in sizes]
    ens = sg.Ensemble([s[0] for s in sizes], [s[1] for s in sizes], [s[2] for s in sizes], params)
    ens.set_engine(engine)
    sims = [sg.Simulation(W, H, n, p) for (W, H, n), p in zip(sizes, params)]
    for j, (W, H, n) in enumerate(sizes):
        agents = agents_uniform(n, W, H, 60.0, 125.0, seed=j)
        ens.upload_agents(j, agents)
        sims[j].upload_agents(agents)
    if tuned:
        ens.autotune(1)
        ens.set_engine(engine)
    ens.prepare_steps(70)
    for k in (70, 20):
        ens.step(k)
    for j, sim in enumerate(sims):
        for _ in range(90):
            sim.step(1)
        assert_bitexact(ens.download_agents(j), sim.download_agents(), f"agents of {j}")
        assert_bitexact(ens.download_trail(j), sim.download_trail(), f"trail of {j}")
    ens.set_reorder(5, 2)
    with pytest.raises(sg.SlimeError):
        ens.step(5)


# Agents, ids and the upload's buffer are 36 bytes an agent, the trails and
# counts 16 a cell, and two arrays of marks one a cell each: not even one of
# them fits, or one.
@pytest.mark.parametrize("spare", [150_000, 420_000])
def test_steps_without_memory_for_marks(gpu, tmp_path, spare):
    import slime_gb300 as sg
    side, n = 512, 20_000
    code = f"""
S, n = {side}, {n}
ens = sg.Ensemble([S], [S], [n], [config0_params(S, S)])
ens.upload_agents(0, agents_uniform(n, S, S, 1.0, 2.0, seed=1))
for m in (3, 20, 20):
    ens.step(m)
np.savez({str(tmp_path / "out.npz")!r}, a=ens.download_agents(0), t=ens.download_trail(0),
         marks=ens.info().marks_colonies, engine=ens.info().engine)
"""
    capped(code, 36 * n + 16 * side * side + spare)
    got = np.load(tmp_path / "out.npz")
    assert got["engine"] == sg.ENSEMBLE_LANES and got["marks"] == 0
    with sg.Simulation(side, side, n, config0_params(side, side)) as sim:
        sim.upload_agents(agents_uniform(n, side, side, 1.0, 2.0, seed=1))
        sim.step(43)
        assert_bitexact(got["a"], sim.download_agents(), "agents")
        assert_bitexact(got["t"], sim.download_trail(), "trail")
