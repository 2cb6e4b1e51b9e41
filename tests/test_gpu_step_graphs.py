"""Calls of the step loop that differ only in what they record share no graph:
a run that wants sample records gets them after a step() of the same dt, and a
step() after such a run appends none."""
import numpy as np
import pytest

from tree_b200 import api, cloud, units

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("precision", [api.PREC_FP64, api.PREC_MIXED])
def test_records_after_calls_without_them(device_lib, precision, graphs):
    c = cloud.make_cloud(200, seed=4)
    dt = units.dt_code(1e-13)
    with api.TreeForce(100, 100, api.Config(physics=api.PHYS_KELBG, precision=precision)) as tf:
        tf.set_graphs(graphs)
        tf.set_state(c.x_el, c.v_el, c.x_ion, c.v_ion)
        assert len(tf.run(dt, 1, 1)) == 1  # the series buffer exists from here on
        tf.step(2 * dt, 1)
        got = tf.run(2 * dt, 1, 1)
        assert list(got["nloop"]) == [3]
        d = tf.step(2 * dt, 1)
        assert list(tf.run(2 * dt, 3, 2)["nloop"]) == [6]
        # the record is that step's
        tf.set_state(c.x_el, c.v_el, c.x_ion, c.v_ion)
        tf.run(dt, 1, 1)
        tf.step(2 * dt, 1)
        again = tf.run(2 * dt, 1, 1)
        np.testing.assert_array_equal(again, got)
        assert np.isfinite([d.epot_e, d.mv2_el]).all()
