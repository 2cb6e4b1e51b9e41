"""A Force call replaces the device positions, so no step follows it without a
new state, whether the call succeeds or fails."""
import numpy as np
import pytest

from tree_b200 import api, cloud, learned_mac, units

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("fails", [False, True])
def test_step_after_force_is_refused(device_lib, learned, fails):
    c = cloud.make_cloud(400, seed=8)
    cfg = api.Config(physics=api.PHYS_KELBG, precision=api.PREC_MIXED,
                     mac=api.MAC_LEARNED if learned else api.MAC_FIXED)
    with api.TreeForce(200, 200, cfg) as tf:
        if learned:
            tf.mac_set_model(*learned_mac.load_model(order=3)[:2])
        tf.set_state(c.x_el, c.v_el, c.x_ion, c.v_ion)
        x = c.x_el.copy()
        if fails:
            x[3, 2] = np.inf
            with pytest.raises(api.TreeGpuError) as e:
                tf.force(x, c.x_ion)
            assert e.value.code == -3
        else:
            tf.force(x, c.x_ion)
        with pytest.raises(api.TreeGpuError) as e:
            tf.step(units.dt_code(1e-13), 1)
        assert e.value.code == -7
