"""An odd number of far cells is evaluated beside a chargeless dummy, which adds
nothing to any target, wherever it lies: here eight targets at +-1e6 um from
their group's centre, and one far cell."""
import numpy as np
import pytest

from tree_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rdf", [False, True])
@pytest.mark.parametrize("order", [2, 3, 4])
def test_one_far_cell_and_a_wide_group(device_lib, order, rdf):
    rng = np.random.default_rng(order)
    corners = np.array([(i, j, k) for i in (-1, 1) for j in (-1, 1) for k in (-1, 1)]) * 1e6
    inside = rng.uniform(-9e5, 9e5, (24, 3))
    far = 3e7 + rng.standard_normal((40, 3)) * 1e4
    x = np.vstack([corners, inside, far])
    el = np.arange(len(x)) % 3 > 0  # the cells are charged
    x_el, x_ion = x[el], x[~el]
    cfg = api.Config(theta=0.5, physics=api.PHYS_KELBG, precision=api.PREC_MIXED)
    bins = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)] if rdf else (None, None)
    with api.TreeForce(len(x_el), len(x_ion), cfg) as tf:
        tf.set_tuning(8, 4, order)
        tf.set_local_expansion(0.0)
        f_el, f_ion, ee, ei = tf.force(x_el, x_ion, *bins)
        t = tf.timings()
        fd, _ = tf.direct(np.arange(len(x)))
    assert t.n_m2p % 2 == 0 and t.n_m2p >= 32  # one cell for the group of 32
    f = np.vstack([f_el, f_ion])
    assert np.isfinite(f).all() and np.isfinite([ee, ei]).all()
    err = np.linalg.norm(f - fd, axis=1) / np.linalg.norm(fd, axis=1)
    assert err.max() < 1e-3
