"""The shared-memory trail tiles at the sizes where they can go wrong: widths
that are not whole 16-byte groups, grids smaller than a tile or than the blur,
every radius, counts and marks; the deposit counts after steps that recorded
marks; the division by nine."""
import ctypes as C

import numpy as np
import pytest

import oracle
from conftest import agents_uniform, config0_params
from test_parity_gpu import assert_bitexact, make_sim


def test_div9_equals_the_division_on_every_input_it_takes():
    assert oracle.div9_mismatches() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tile", range(1, 8))
@pytest.mark.parametrize("W,H", [(131, 67), (260, 65), (3, 5), (1, 1), (64, 8), (129, 130)])
def test_tiles_bitexact(gpu, tile, W, H):
    n = 3000
    rng = np.random.default_rng(W + tile)
    for blur_mode, radius in ((0, 1.0), (1, 0.0), (1, 1.0), (1, 2.0), (1, 4.0), (1, 5.0), (1, 8.0)):
        for exact_counts, dep in ((0, 1.0), (1, 0.3)):
            p = config0_params(W, H, decay_mode=blur_mode, decay_factor=0.97 if blur_mode else 10.0, blur_mode=blur_mode,
                               blur_radius=radius, blur_sigma=1.7, pheromone_deposition_amount=dep)
            agents = agents_uniform(n, W, H, 1.0, 2.0, seed=4)
            trail = rng.random((H, W), dtype=np.float32)
            sim = make_sim(W, H, n, p, agents, trail)
            sim.set_options(trail_tile=tile, exact_counts=exact_counts)
            sim.step(2)
            ca, ct = agents.copy(), trail.copy()
            oracle.run(p, W, H, ca, ct, 2)
            what = f"{W}x{H} tile {tile} blur {blur_mode} r {radius} dep {dep}"
            assert_bitexact(sim.download_trail(), ct, "trail " + what)
            assert_bitexact(sim.download_agents(), ca, "agents " + what)
            sim.close()


@pytest.mark.gpu
def test_box_of_tiny_huge_and_special_values(gpu):
    """Sums outside the range of the division-free average: subnormal, huge,
    infinite and NaN cells."""
    W, H = 132, 40
    rng = np.random.default_rng(1)
    trail = (rng.random((H, W)) * 10.0 ** rng.uniform(-46, 38, (H, W))).astype(np.float32)
    trail[3, 5], trail[30, 100], trail[9, :] = np.inf, np.nan, 0.0
    p = config0_params(W, H, decay_mode=1, decay_factor=1.0, blur_mode=0, diffusion_rate=1.0)
    for tile in (1, 4, 8, 10):
        sim = make_sim(W, H, 0, p, np.zeros((0, 4), np.float32), trail)
        sim.set_options(trail_tile=tile)
        sim.step(1)
        ca, ct = np.zeros((0, 4), np.float32), trail.copy()
        oracle.run(p, W, H, ca, ct, 1)
        got = sim.download_trail()
        assert np.array_equal(np.isnan(got), np.isnan(ct))
        assert_bitexact(got[~np.isnan(ct)], ct[~np.isnan(ct)], f"tile {tile}")


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,dispatch", [(200, 96, 0), (203, 96, 0), (200, 96, 1)])
def test_counts_after_steps_that_recorded_marks(gpu, W, H, dispatch):
    """A context that neither chose nor tuned a tile keeps giving the last
    step's counts, also after the agents were replaced."""
    n = 9000 if not dispatch else 4_264_240
    p = config0_params(W, H, dispatch_mode=dispatch)
    agents = agents_uniform(n, W, H, 1.0, 2.0, seed=8)
    trail = np.random.default_rng(9).random((H, W), dtype=np.float32)
    sim = make_sim(W, H, n, p, agents, trail)
    ca, ct = agents.copy(), trail.copy()
    want = oracle.run(p, W, H, ca, ct, 2, record_counts=True)[-1]
    sim.step(2)
    assert_bitexact(sim.download_deposit_counts(), want, "counts")
    ca2, ct2 = ca.copy(), ct.copy()
    want = oracle.run(p, W, H, ca2, ct2, 1, record_counts=True)[-1]
    sim.step(1)
    sim.reorder_agents()
    sim.upload_agents(agents)
    assert_bitexact(sim.download_deposit_counts(), want, "counts after an upload")
    # steps that count and steps that mark, in turn
    a, t = agents.copy(), ct2.copy()
    for exact in (1, 0, 1):
        sim.set_options(exact_counts=exact)
        sim.step(1)
        want = oracle.run(p, W, H, a, t, 1, record_counts=True)[-1]
        assert_bitexact(sim.download_deposit_counts(), want, f"counts, exact {exact}")
        assert_bitexact(sim.download_trail(), t, f"trail, exact {exact}")


@pytest.mark.gpu
def test_caller_buffers_of_any_alignment(gpu):
    """The caller-owned step with trails and counts off the 16-byte grid."""
    import torch

    import slime_gb300 as sg
    W, H, n = 128, 50, 3001
    p = config0_params(W, H, blur_mode=0, decay_mode=0, decay_factor=10.0)
    agents = agents_uniform(n, W, H, 1.0, 2.0, seed=2)
    trail = np.random.default_rng(3).random((H, W), dtype=np.float32)
    ca, ct = agents.copy(), trail.copy()
    oracle.run(p, W, H, ca, ct, 1)

    def at(offset, values):
        buf = torch.zeros(values.size + 8, device="cuda", dtype=torch.float32)
        v = buf[offset:offset + values.size]
        v.copy_(torch.from_numpy(np.ascontiguousarray(values, np.float32).reshape(-1)))
        return v

    ptr = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
    for offsets in ((0,) * 7, (1, 2, 3, 1, 1, 2, 3), (0, 0, 0, 0, 0, 2, 0), (1, 1, 1, 1, 0, 0, 0)):
        cols = [at(offsets[j], agents[:, j]) for j in range(4)]
        src, dst, counts = at(offsets[4], trail), at(offsets[5], trail * 0), at(offsets[6], trail * 0)
        rc = sg.lib().slime_step_noalloc_scratch(C.byref(p), W, H, n, *[ptr(c) for c in cols], ptr(src), ptr(dst),
                                                 ptr(counts), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        torch.cuda.synchronize()
        assert_bitexact(dst.cpu().numpy().reshape(H, W), ct, f"trail at {offsets}")
        assert_bitexact(torch.stack(cols, 1).cpu().numpy(), ca, f"agents at {offsets}")
