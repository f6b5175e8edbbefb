"""Performance cases of the Physarum core: what its users have it do, through its public entry points.

A case is a dict of plain values; its "kind" says which entry points the pass goes through:

  run       Simulation.step(n), then the agents and the trail read back into host arrays the program keeps
  frame     one frame of a display loop: the parameter block, one step, the colourised image on the host
  scratch   slime_step_noalloc_scratch on device buffers the caller owns (torch tensors here)
  noalloc   slime_step_noalloc, the same with the library's own count array (trails up to 1,048,576 cells)
  adjoint   trail_chain forward and backward: a training step on the trail parameters
  ensemble  Ensemble.step(n) over colonies of uneven sizes, then every colony read back

"tuned" is whether the program calls autotune() once, as the benchmark does; "reorder" is its
options.reorder_every.  Passes continue from the state the pass before left, as a running program does.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "slime-mold_gb300"))

import slime_gb300 as sg  # noqa: E402
from slime_gb300.autograd import trail_chain  # noqa: E402

PLAIN = "plain"  # params(): the benchmark's parameters instead of a preset's


def listed():
    return [
        # A small colony shown live: 512^2, one frame per call. Latency and launches are all there is.
        dict(name="frame 512", kind="frame", width=512, height=512, agents=65_536, params=PLAIN, blur=1, sensor=9.0,
             speed=1.0, jitter=0.05, deposition=1.0, reorder=0, tuned=False, image_w=512, image_h=512),
        # The 512^2 configuration run for its 100 steps at a time, tuned.
        dict(name="run 512", kind="run", width=512, height=512, agents=65_536, params=PLAIN, blur=1, sensor=9.0,
             speed=1.0, jitter=0.05, deposition=1.0, reorder=200, tuned=True, steps=100),
        # The reference application's own frame: its default settings, 10 M agents on its 1600x900 window.
        dict(name="frame app 1600x900", kind="frame", width=1600, height=900, agents=10_000_000, params="Default", blur=0,
             reorder=0, tuned=False, image_w=1600, image_h=900),
        # The integration guide's first program: a preset, seeded, 100 steps, default options, the trail back.
        dict(name="run app 1600x900", kind="run", width=1600, height=900, agents=10_000_000, params="Sponge", blur=0,
             reorder=0, tuned=False, steps=100),
        # An odd window dragged to some size: rows of no alignment, agents of no round number.
        dict(name="run odd 1001x777", kind="run", width=1001, height=777, agents=500_003, params="Waves", blur=0,
             reorder=0, tuned=False, steps=100),
        # A wide Gaussian (the blur option up to radius 8) on a medium trail, tuned.
        dict(name="run blur5 2048", kind="run", width=2048, height=2048, agents=1_048_576, params=PLAIN, blur=5, sensor=9.0,
             speed=1.0, jitter=0.05, deposition=1.0, reorder=200, tuned=True, steps=100),
        # The benchmark's workload: 16.8 M agents on 4096^2, Morton reorder every 200 steps, tuned.
        dict(name="run 4096", kind="run", width=4096, height=4096, agents=16_777_216, params=PLAIN, blur=1, sensor=9.0,
             speed=1.0, jitter=0.05, deposition=1.0, reorder=200, tuned=True, steps=200),
        # The largest configuration: 67 M agents on 8192^2, reordered every 50 steps, tuned.
        dict(name="run 8192", kind="run", width=8192, height=8192, agents=67_108_864, params=PLAIN, blur=1, sensor=18.0,
             speed=1.5, jitter=0.05, deposition=1.0, reorder=50, tuned=True, steps=100),
        # A host engine that owns all device memory steps a 1024^2 colony in its own buffers.
        dict(name="noalloc 1024", kind="noalloc", width=1024, height=1024, agents=1_048_576, params=PLAIN, blur=1, sensor=9.0,
             speed=1.0, jitter=0.05, deposition=1.0),
        # The same with its own count array, a larger odd trail and a deposition that does not saturate.
        dict(name="scratch odd 3001x2003", kind="scratch", width=3001, height=2003, agents=4_000_037, params="Default",
             blur=0, deposition=0.3),
        # A training step on decay, diffusion and deposition: 1024^2, 200 steps, checkpoints every 50.
        dict(name="adjoint 1024", kind="adjoint", width=1024, height=1024, agents=1_048_576, params=PLAIN, blur=1, sensor=9.0,
             speed=1.0, jitter=0.05, deposition=1e-4, decay=0.95, steps=200, every=50),
        # A parameter sweep: 16 colonies of 256^2 to 1024^2 at 0.25 to 4 agents per cell, tuned.
        dict(name="ensemble 16", kind="ensemble", colonies=16, side_log2_lo=8, side_log2_hi=10, colony_seed=1, reorder=200,
             tuned=True, steps=100),
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _side(rng, lo, hi, odd):
    s = _between(rng, lo, hi)
    return s | 1 if odd else max(lo, s // 4 * 4)


def draw(rng):
    kind = rng.choice(["run", "run", "run", "frame", "noalloc", "scratch", "adjoint", "ensemble"])
    if kind == "ensemble":
        return dict(kind=kind, colonies=_between(rng, 2, 24), side_log2_lo=rng.randint(7, 8),
                    side_log2_hi=rng.randint(9, 10), colony_seed=rng.randrange(1 << 20), reorder=rng.choice([0, 200]),
                    tuned=rng.random() < 0.7, steps=_between(rng, 20, 100))
    odd = rng.random() < 0.35
    top = {"run": 4096, "frame": 2048, "noalloc": 1000, "scratch": 4096, "adjoint": 1400}[kind]
    c = dict(kind=kind, width=_side(rng, 256, top, odd), height=_side(rng, 256, top, rng.random() < 0.35))
    cells = c["width"] * c["height"]
    c["agents"] = max(1000, min(20_000_000, int(cells * math.exp(rng.uniform(math.log(0.1), math.log(6.0))))))
    c["params"] = rng.choice([PLAIN, "Default", "Sponge", "Firecracker Trees", "Threads", "Waves", "Snake"])
    c["blur"] = rng.choice([1, 1, 2, 3, 5, 8]) if c["params"] == PLAIN else 0
    if c["params"] == PLAIN or kind == "adjoint":
        c["params"] = PLAIN
        c["blur"] = c["blur"] or rng.choice([0, 1])
        c.update(sensor=round(rng.uniform(4.0, 20.0), 3), speed=round(rng.uniform(1.0, 40.0), 3),
                 jitter=rng.choice([0.0, 0.05, 0.1]), deposition=rng.choice([1.0, 1.0, round(rng.uniform(0.2, 2.0), 3)]))
    if kind == "run":
        c.update(reorder=rng.choice([0, 50, 200]), tuned=rng.random() < 0.6, steps=_between(rng, 10, 200))
        # a draw costs no more than the largest listed case, unsorted agents included
        c["steps"] = max(10, min(c["steps"], int(1.2e9 / (c["agents"] + cells / 4))))
    elif kind == "frame":
        c.update(reorder=rng.choice([0, 200]), tuned=rng.random() < 0.4, image_w=_between(rng, 320, 1920),
                 image_h=_between(rng, 240, 1200))
    elif kind == "adjoint":
        c.update(deposition=rng.choice([1e-4, 1.0]), decay=round(rng.uniform(0.9, 0.97), 4),
                 steps=_between(rng, 30, 200), every=rng.choice([25, 50]))
    return c


# ---------------------------------------------------------------------------------------------- parameters
def _params(case, width=None, height=None):
    W, H = width or case["width"], height or case["height"]
    if case["params"] == PLAIN:
        p = sg.SlimeParams()
        p.width, p.height = W, H
        p.decay_factor = case.get("decay", 0.97)
        p.agent_jitter = case["jitter"]
        p.agent_speed_min, p.agent_speed_max = case["speed"], 2.0 * case["speed"]
        p.agent_turn_speed = 0.3
        p.agent_sensor_angle = 0.4
        p.agent_sensor_distance = case["sensor"]
        p.diffusion_rate = 0.5
        p.time_step = 0.016
        p.decay_mode = sg.DECAY_MULTIPLY
        p.blur_mode = sg.BLUR_GAUSS if case["blur"] else sg.BLUR_REF_BOX3
        p.blur_radius = float(case["blur"])
        p.blur_sigma = max(1.0, 0.4 * case["blur"])
    else:
        p = sg.params_from_settings(sg.preset(case["params"]), W, H)
    if "deposition" in case:
        p.pheromone_deposition_amount = case["deposition"]
    return p


def _headings(case):
    """The reference draws a preset's headings from 0..360; the benchmark from a full turn."""
    return (0.0, 2.0 * math.pi) if case["params"] == PLAIN else (0.0, 360.0)


def _host(shape, dtype=torch.float32):
    """Page-locked host memory, as a program that reads back again and again keeps it."""
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _uniform(gen, n, lo, hi):
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float32) * (hi - lo) + lo
    return torch.minimum(u, torch.nextafter(torch.full((), hi, device="cuda"), torch.zeros((), device="cuda")))


def _inputs(case, seed):
    """x, y, angle, speed and trail on the GPU: agents anywhere, a trail that has cells of 0 and of nearly 1."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    W, H, n, p = case["width"], case["height"], case["agents"], _params(case)
    h0, h1 = _headings(case)
    cols = [_uniform(gen, n, 0.0, float(W)), _uniform(gen, n, 0.0, float(H)), _uniform(gen, n, h0, h1),
            torch.rand(n, generator=gen, device="cuda") * (p.agent_speed_max - p.agent_speed_min) + p.agent_speed_min]
    trail = torch.rand((H, W), generator=gen, device="cuda")
    trail = trail * (torch.rand((H, W), generator=gen, device="cuda") < 0.6)
    return cols, trail


def _lut():
    i = np.arange(256)
    return np.concatenate([i, 255 - i, (i * 7) % 256]).astype(np.uint8)


# ---------------------------------------------------------------------------------------------- the passes
def _colonies(case):
    rng = np.random.default_rng(case["colony_seed"])
    out = []
    for _ in range(case["colonies"]):
        side = 1 << int(rng.integers(case["side_log2_lo"], case["side_log2_hi"] + 1))
        p = sg.SlimeParams()
        p.width, p.height = side, side
        p.decay_factor = float(rng.uniform(0.90, 0.995))
        p.agent_jitter = float(rng.uniform(0.0, 0.1))
        p.agent_speed_min, p.agent_speed_max = 1.0, 2.0
        p.agent_turn_speed = float(rng.uniform(0.1, 0.6))
        p.agent_sensor_angle = float(rng.uniform(0.2, 0.8))
        p.agent_sensor_distance = float(rng.uniform(4, 20))
        p.diffusion_rate = float(rng.uniform(0.1, 0.9))
        p.pheromone_deposition_amount = float(rng.uniform(0.5, 2.0))
        p.blur_radius = p.blur_sigma = 1.0
        p.time_step = 0.016
        p.decay_mode, p.blur_mode = sg.DECAY_MULTIPLY, sg.BLUR_GAUSS
        out.append((side, int(side * side * rng.uniform(0.25, 4.0)), p))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "ensemble":
        cols = _colonies(case)
        sides = [c[0] for c in cols]
        e = sg.Ensemble(sides, sides, [c[1] for c in cols], [c[2] for c in cols])
        for j in range(len(cols)):
            e.seed_agents(j, seed * 1000 + j)
        e.set_reorder(case["reorder"], 2)
        if case["tuned"]:
            e.autotune(2)
        s["ensemble"] = e
        return s
    W, H, n = case["width"], case["height"], case["agents"]
    p = s["params"] = _params(case)
    if kind in ("noalloc", "scratch"):
        s["cols"], a = _inputs(case, seed)
        s["trails"] = [a, torch.empty_like(a)]
        if kind == "scratch":
            s["counts"] = torch.empty((H, W), dtype=torch.int32, device="cuda")
        return s
    s["sim"] = sim = sg.Simulation(W, H, n, p)
    if kind == "adjoint":
        cols, trail = _inputs(case, seed)
        s["agents"] = torch.stack(cols, dim=1).cpu().numpy()
        s["trail0"] = (trail * 0.3 + 0.01).cpu()
        gen = torch.Generator().manual_seed(seed)
        s["weight"] = torch.rand((H, W), generator=gen)
        return s
    sim.seed_agents(seed, *_headings(case))
    sim.set_options(reorder_every=case["reorder"])
    if case["tuned"]:
        sim.autotune()
    if kind == "run":
        s["agents"], s["trail"] = _host((n, 4)), _host((H, W))
    else:
        s["image"] = _host((case["image_h"], case["image_w"], 4), torch.uint8)
        s["lut"] = _lut()
    return s


def _run_noalloc(s):
    c, L = s["case"], sg.lib()
    src, dst = s["trails"]
    at = [ctypes.c_void_p(t.data_ptr()) for t in (*s["cols"], src, dst)]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if c["kind"] == "noalloc":
        rc = L.slime_step_noalloc(ctypes.byref(s["params"]), c["width"], c["height"], c["agents"], *at, stream)
    else:
        rc = L.slime_step_noalloc_scratch(ctypes.byref(s["params"]), c["width"], c["height"], c["agents"], *at,
                                          ctypes.c_void_p(s["counts"].data_ptr()), stream)
    if rc != 0:
        raise RuntimeError(f"{c['kind']} step: status {rc}")
    s["trails"] = [dst, src]
    x, y, angle, speed = s["cols"]
    return {"x": x, "y": y, "angle": angle, "speed": speed, "trail": dst}


def _run_adjoint(s):
    c, p = s["case"], s["params"]
    trail0 = s["trail0"].clone().requires_grad_()
    decay = torch.tensor(p.decay_factor, requires_grad=True)
    rate = torch.tensor(p.diffusion_rate, requires_grad=True)
    deposition = torch.tensor(p.pheromone_deposition_amount, requires_grad=True)
    out = trail_chain(trail0, decay, rate, deposition, s["sim"], c["steps"], c["every"], s["agents"])
    (out * s["weight"]).sum().backward()
    return {"trail": out.detach(), "d_trail0": trail0.grad, "d_decay": decay.grad, "d_rate": rate.grad,
            "d_deposition": deposition.grad}


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind in ("noalloc", "scratch"):
        return _run_noalloc(s)
    if kind == "adjoint":
        return _run_adjoint(s)
    if kind == "ensemble":
        e = s["ensemble"]
        e.step(c["steps"])
        return [{"agents": e.download_agents(j), "trail": e.download_trail(j)} for j in range(c["colonies"])]
    sim = s["sim"]
    if kind == "frame":
        sim.set_params(s["params"])
        sim.step(1)
        sim.colorize_async(s["lut"], s["image"])
        sim.wait_download()
        return s["image"]
    sim.step(c["steps"])
    return {"agents": sim.download_agents(s["agents"]), "trail": sim.download_trail(s["trail"])}


# ---------------------------------------------------------------------------------------------- the work
AGENT_FLOPS = 200  # five sines and cosines, three bilinear samples, turn, move and wrap
CELL_FLOPS = 20    # fold, decay and a separable 3x3 blur


def work(case):
    """Per step: every agent's state read and written once (32 B), every cell read and written once (8 B)."""
    kind = case["kind"]
    if kind == "ensemble":
        cols = _colonies(case)
        n, cells = sum(c[1] for c in cols), sum(c[0] * c[0] for c in cols)
    else:
        n, cells = case["agents"], case["width"] * case["height"]
    steps = case.get("steps", 1)
    cell_flops = CELL_FLOPS + 8 * max(0, case.get("blur", 0) - 1)
    b, f = steps * (32 * n + 8 * cells), steps * (AGENT_FLOPS * n + cell_flops * cells)
    if kind == "run":
        b += 16 * n + 4 * cells  # read back
    elif kind == "ensemble":
        b += 16 * n + 4 * cells
    elif kind == "frame":
        b += 4 * case["image_w"] * case["image_h"]
    elif kind == "adjoint":
        # backward: per step the recorded trail and deposit counts and dL/dT read, dL/dT written; the agents of
        # a segment replayed once (the counts of all steps are not kept)
        b += steps * (16 * cells + 32 * n)
        f += steps * (2 * cell_flops * cells + AGENT_FLOPS * n)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------------- 64-bit values
def _f32(x):
    return float(np.float32(x))


def _mix(a, b, t):
    return a * (1 - t) + b * t


def _blur64(t, p):
    if p.blur_mode == sg.BLUR_GAUSS:
        r = int(p.blur_radius)
        w = torch.tensor([math.exp(-i * i / (2.0 * p.blur_sigma * p.blur_sigma)) for i in range(-r, r + 1)],
                         dtype=torch.float64, device=t.device)
        w = w / w.sum()
        for dim in (0, 1):
            t = sum(w[i + r] * torch.roll(t, i, dim) for i in range(-r, r + 1))
        return t
    return sum(torch.roll(t, (i, j), (0, 1)) for i in (-1, 0, 1) for j in (-1, 0, 1)) / 9.0


def _sample64(trail, x, y):
    H, W = trail.shape
    x0, y0 = torch.floor(x), torch.floor(y)
    ok = (x0 >= 0) & (x0 + 1 < W) & (y0 >= 0) & (y0 + 1 < H)
    xi, yi = torch.where(ok, x0, 0).long(), torch.where(ok, y0, 0).long()
    dx, dy = x - x0, y - y0
    at = lambda i, j: trail[torch.clamp(yi + j, max=H - 1), torch.clamp(xi + i, max=W - 1)]  # noqa: E731
    v = _mix(_mix(at(0, 0), at(1, 0), dx), _mix(at(0, 1), at(1, 1), dx), dy)
    return torch.where(ok, v, 0.0)


def _step64(case, seed):
    """One step from prepare()'s inputs in 64 bits. The jitter hash is defined on the 32-bit value of its argument
    (index, x and y rounded as the shader's f32 arithmetic rounds them); its sine is taken in 64 bits."""
    cols, trail32 = _inputs(case, seed)
    p = _params(case)
    W, H, n = case["width"], case["height"], case["agents"]
    x, y, th, v = (c.double() for c in cols)
    trail = trail32.double()
    v = torch.clamp(v, p.agent_speed_min, p.agent_speed_max)
    d, a = p.agent_sensor_distance, p.agent_sensor_angle
    left, right, center = (_sample64(trail, x + d * torch.cos(t), y + d * torch.sin(t)) for t in (th - a, th + a, th))
    straight = (center > left) & (center > right)
    go_l, go_r = ~straight & (left > right), ~straight & (right > left)
    tau = 6.28318530718
    turn = min(p.agent_turn_speed, tau)
    th = th + turn * (go_r.double() - go_l.double())
    arg = torch.arange(n, device="cuda", dtype=torch.int32).float() * _f32(12.9898)
    arg = arg + cols[0] * _f32(78.233)
    arg = arg + cols[1] * _f32(37.719)
    h = torch.sin(arg.double()) * _f32(43758.5453)
    th = th + ((h - torch.floor(h)) * 2 - 1) * p.agent_jitter
    th = torch.fmod(th, tau)
    th = torch.where(th < 0, th + tau, th)
    x = torch.fmod(x + v * p.time_step * torch.cos(th), W)
    y = torch.fmod(y + v * p.time_step * torch.sin(th), H)
    x, y = torch.where(x < 0, x + W, x), torch.where(y < 0, y + H, y)
    cell = torch.clamp(y.long(), max=H - 1) * W + torch.clamp(x.long(), max=W - 1)
    k = torch.bincount(cell, minlength=W * H).reshape(H, W).double()
    t = torch.where(k > 0, torch.clamp(trail + k * p.pheromone_deposition_amount, 0, 1), trail)
    t = t * p.decay_factor if p.decay_mode == sg.DECAY_MULTIPLY else torch.clamp(t - p.decay_factor * 0.001, min=0)
    rate = min(max(p.diffusion_rate, 0.0), 1.0)
    return {"x": x, "y": y, "angle": th, "speed": v, "trail": _mix(t, _blur64(t, p), rate)}


def exact(case, seed):
    """The allocation-free steps (one step from given inputs). Runs of many steps have no such value: each agent's
    jitter hashes the bits of its position, so 32 and 64 bits part after a step or two. Of the adjoint, dL/dT0 where
    no deposit saturates: the chain is then linear in the trail, whatever the trajectories."""
    if case["kind"] in ("noalloc", "scratch"):
        return _step64(case, seed)
    if case["kind"] == "adjoint" and case["deposition"] <= 1e-4:
        p = _params(case)
        gen = torch.Generator().manual_seed(seed)
        g = torch.rand((case["height"], case["width"]), generator=gen).cuda().double()
        for _ in range(case["steps"]):
            g = p.decay_factor * _mix(g, _blur64(g, p), p.diffusion_rate)
        return {"trail": None, "d_trail0": g, "d_decay": None, "d_rate": None, "d_deposition": None}
    return None
