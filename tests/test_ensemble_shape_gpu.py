"""The cooperative launch shape chosen by hand is the one that steps, unless
the engine was chosen or tuned."""
import pytest

from conftest import config0_params

pytestmark = pytest.mark.gpu


def test_a_shape_by_hand_steps_cooperatively(gpu):
    import slime_gb300 as sg

    def ensemble():
        return sg.Ensemble([64, 128], [32, 64], [500, 3000], [config0_params(64, 32), config0_params(128, 64)])

    ens = ensemble()
    ens.set_shape(16, 2, 2)
    assert ens.info().engine == sg.ENSEMBLE_COOPERATIVE
    before = ens.launch_count()
    ens.step(7)
    assert ens.launch_count() - before == 7  # one launch a step
    ens = ensemble()
    ens.set_engine(sg.ENSEMBLE_LANES)
    ens.set_shape(16, 2, 2)
    assert ens.info().engine == sg.ENSEMBLE_LANES
    ens = ensemble()
    ens.autotune(1)
    tuned = ens.info().engine
    ens.set_shape(16, 2, 2)
    assert ens.info().engine == tuned
