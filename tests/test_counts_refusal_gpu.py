"""The refusal of deposit counts says why they are refused, whatever the step
recorded: marks (one agent per cell and fewer) or counts (more)."""
import pytest

from conftest import agents_uniform, config0_params
from test_parity_gpu import STREAM8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 30_000])
def test_the_refusal_names_its_reason(gpu, n):
    import slime_gb300 as sg
    W, H = 128, 96  # 12,288 cells
    with sg.Simulation(W, H, n, config0_params(W, H)) as sim:
        sim.upload_agents(agents_uniform(n, W, H, 1.0, 2.0))
        sim.set_options(trail_tile=STREAM8)
        sim.step(1)
        with pytest.raises(sg.SlimeError) as refused:
            sim.download_deposit_counts()
        assert refused.value.status == -4  # SLIME_ERR_STATE
        assert "streaming trail tile" in str(refused.value) and "exact_counts" in str(refused.value)
        assert "not how many" not in str(refused.value)
        sim.set_options(trail_tile=STREAM8, exact_counts=1)
        sim.step(1)
        assert sim.download_deposit_counts().sum() > 0
