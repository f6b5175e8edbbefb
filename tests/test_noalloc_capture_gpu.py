"""slime_step_noalloc and slime_step_noalloc_scratch inside a caller's stream
capture: the count clear, the agent pass and the trail pass are graph nodes
joined by programmatic edges, and replays of the graph step as the calls do."""
import ctypes as C

import numpy as np
import pytest

from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim

pytestmark = pytest.mark.gpu


def _ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("scratch", [False, True])
@pytest.mark.parametrize("W,H,dispatch,dep", [(320, 200, 0, 1.0), (131, 77, 0, 0.3), (320, 200, 1, 0.3)])
def test_captured_steps(gpu, scratch, W, H, dispatch, dep):
    import torch

    import slime_gb300 as sg
    L = sg.lib()
    n, replays = (30_001 if not dispatch else 4_264_240), 3
    p = config0_params(W, H, agent_speed_min=30.0, agent_speed_max=50.0, agent_jitter=0.3, dispatch_mode=dispatch,
                       pheromone_deposition_amount=dep)
    agents = agents_uniform(n, W, H, 30.0, 50.0, seed=5)
    trail = np.random.default_rng(6).random((H, W), dtype=np.float32)
    dev = torch.device("cuda", 0)
    cols = [torch.tensor(np.ascontiguousarray(agents[:, j]), device=dev) for j in range(4)]
    ta = torch.tensor(trail, device=dev)
    tb = torch.empty_like(ta)
    counts = torch.full((H * W,), 7, dtype=torch.int32, device=dev)

    def step(src, dst, stream):
        args = [C.byref(p), W, H, n, *[_ptr(c) for c in cols], _ptr(src), _ptr(dst)]
        s = C.c_void_p(stream.cuda_stream)
        rc = L.slime_step_noalloc_scratch(*args, _ptr(counts), s) if scratch else L.slime_step_noalloc(*args, s)
        assert rc == 0

    keep = [c.clone() for c in cols]
    warm = torch.cuda.Stream()
    with torch.cuda.stream(warm):  # the library's module is loaded before the capture
        step(ta, tb, warm)
    torch.cuda.synchronize()
    for c, k in zip(cols, keep):
        c.copy_(k)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s = torch.cuda.current_stream()
        step(ta, tb, s)
        tb.mul_(1.0)  # a kernel of the caller's between the steps
        step(tb, ta, s)
    torch.cuda.synchronize()
    for _ in range(replays):
        g.replay()
    torch.cuda.synchronize()
    with make_sim(W, H, n, p, agents, trail) as sim:
        for _ in range(2 * replays):
            sim.step(1)
        assert_bitexact(np.stack([c.cpu().numpy() for c in cols], axis=1), sim.download_agents(), "agents")
        assert_bitexact(ta.cpu().numpy(), sim.download_trail(), "trail")
