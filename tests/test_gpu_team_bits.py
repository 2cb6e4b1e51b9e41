"""Teams of every size give one warp's bits, under both pair laws: a cloud alone
(its own size of team) and inside an ensemble large enough for one warp per
group."""
import numpy as np
import pytest

from tree_b200 import api, cloud, learned_mac, units

pytestmark = pytest.mark.gpu

SIZES = [(700, 699), (2100, 2101), (5000, 5001), (12500, 12500)]  # teams of 16, 8, 4, 2


@pytest.mark.parametrize("learned,order", [(False, 2), (False, 3), (False, 4), (True, 3),
                                           (True, 4)])  # no model of the quadrupole
@pytest.mark.parametrize("physics", [api.PHYS_REF, api.PHYS_KELBG])
def test_alone_and_in_an_ensemble(device_lib, learned, physics, order):
    dt = units.dt_code(1e-13)
    cl = []
    for n_el, n_ion in SIZES:
        c = cloud.make_cloud(2 * max(n_el, n_ion), seed=n_el)
        rng = np.random.Generator(np.random.Philox(n_ion))
        cl.append((c.x_ion[:n_el] + rng.standard_normal((n_el, 3)) * 0.3, c.x_ion[:n_ion]))
    cfg = api.Config(theta=0.42, physics=physics, precision=api.PREC_MIXED,
                     mac=api.MAC_LEARNED if learned else api.MAC_FIXED)

    def tuned(tf):
        tf.set_tuning(8, 4, order)
        if learned:
            tf.mac_set_model(*learned_mac.load_model(order=order)[:2])
            tf.mac_config(3e-5, 0.05, 0.9)
        return tf

    x = np.vstack([np.vstack(c) for c in cl])
    assert len(x) >= 30000
    with tuned(api.Ensemble([cfg] * len(cl), *zip(*SIZES))) as ens:
        ens.set_state(x, np.zeros_like(x))
        ens.step(dt, 1)
        fe = ens.get_state()["f"]
        for k, (c, s) in enumerate(zip(cl, SIZES)):
            with tuned(api.TreeForce(*s, cfg)) as tf:
                tf.set_state(c[0], np.zeros_like(c[0]), c[1], np.zeros_like(c[1]))
                tf.step(dt, 1)
                st = tf.get_state()
            np.testing.assert_array_equal(fe[ens.offsets[k]:ens.offsets[k + 1]],
                                          np.vstack([st["f_el"], st["f_ion"]]))
