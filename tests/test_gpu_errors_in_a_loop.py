"""An error in any step of a call is the call's: a step whose tree did not fit
leaves the forces of the step before it, so the call fails although the steps
after it succeed; the nodes have grown by then, and the call made again from
reloaded state gives what a handle with room from the start gives."""
import numpy as np
import pytest

from tree_b200 import api

pytestmark = pytest.mark.gpu

DT = 1e-3


def _state(n):
    """At the first step every two electrons are 1e-9 um apart (about 30 tree
    levels of their own), before and after it 0.5 um."""
    rng = np.random.default_rng(n)
    x_ion = rng.standard_normal((n, 3)) * 20.0
    met = rng.standard_normal((n // 2, 3)) * 20.0
    met = np.repeat(met, 2, axis=0)
    met[1::2] += 1e-9
    v = rng.standard_normal((n // 2, 3))
    v *= 0.25 / DT / np.linalg.norm(v, axis=1, keepdims=True)
    v_el = np.empty_like(met)
    v_el[0::2], v_el[1::2] = v, -v
    zero = np.zeros((n, 3))
    return met - DT * v_el, v_el, zero, x_ion, zero, zero


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("precision", [api.PREC_FP64, api.PREC_MIXED])
@pytest.mark.parametrize("n", [1000, 10000])
def test_first_of_two_steps_does_not_fit(device_lib, n, precision, graphs):
    st = _state(n)
    cfg = api.Config(physics=api.PHYS_KELBG, precision=precision)
    with api.TreeForce(n, n, cfg) as tf, api.TreeForce(n, n, cfg) as roomy:
        tf.set_graphs(graphs)
        tf.load_state(*st)
        tf.step(1e-9, 1)  # far apart: the tree fits
        tf.load_state(*st)
        with pytest.raises(api.TreeGpuError) as e:
            tf.step(DT, 2)
        assert e.value.code == -4
        tf.load_state(*st)
        tf.step(DT, 2)
        roomy.set_state(st[0] + DT * st[1], st[1], st[3], st[4])  # grows for this tree
        roomy.load_state(*st)
        roomy.step(DT, 2)
        for k, v in roomy.get_state().items():
            np.testing.assert_array_equal(tf.get_state()[k], v)


@pytest.mark.parametrize("precision", [api.PREC_FP64, api.PREC_MIXED])
def test_an_error_is_reported_once(device_lib, precision):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((200, 3))
    bad = x.copy()
    bad[5, 1] = np.nan
    with api.TreeForce(100, 100, api.Config(physics=api.PHYS_KELBG, precision=precision)) as tf:
        for _ in range(2):
            want = tf.force(x[:100], x[100:])[0]
            with pytest.raises(api.TreeGpuError) as e:
                tf.force(bad[:100], bad[100:])
            assert e.value.code == -3
            np.testing.assert_array_equal(tf.force(x[:100], x[100:])[0], want)
