"""Which uploaded trails may take deposit marks, at sizes on both sides of where
the device looks at the values instead of the host: seen by whether a marking
tile can still say the exact counts.  A single bad value at either end or
between must be found; zeros of both signs and +inf are fine."""
import numpy as np
import pytest

from conftest import agents_uniform, config0_params
from test_parity_gpu import STREAM8, make_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(64, 5), (60, 1092), (256, 256), (1028, 333), (2048, 1500)])  # 65,520 and 65,536 cells
@pytest.mark.parametrize("value,marks", [(np.nan, False), (-1e-45, False), (-np.inf, False), (-0.0, True), (np.inf, True)])
def test_one_value_decides(gpu, W, H, value, marks):
    n = 200
    sim = make_sim(W, H, n, config0_params(W, H), agents_uniform(n, W, H, 1.0, 2.0, seed=1),
                   np.zeros((H, W), np.float32))
    sim.set_options(trail_tile=STREAM8)
    for at in (0, W * H // 2 + 1, W * H - 1):
        trail = np.full((H, W), 0.25, np.float32)
        trail.flat[at] = value
        sim.upload_trail(trail)
        sim.step(1)
        if marks:
            with pytest.raises(RuntimeError):
                sim.download_deposit_counts()
        else:
            assert sim.download_deposit_counts().sum() == n
