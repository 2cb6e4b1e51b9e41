"""The direct sum decides on the reference laws' cutoff (like charges within
r^2 <= 0.01 contribute nothing) as the reference forms r^2, also where a sum with
fused operations falls on the other side of it."""
import numpy as np
import pytest

import oracle
from tree_b200 import api, units

pytestmark = pytest.mark.gpu

# offsets whose (x^2 + y^2) + z^2 is at most 0.01 while the fused sum is above,
# then the other way round
TIES = [
    (0.02626478913657202, 0.014553650572524475, 0.09538528244244113),
    (0.011957819004532425, 0.02354424800174388, 0.09645039632208477),
    (0.048070575100403426, 0.041232379910798436, 0.07738934459218569),
    (0.0668037383667878, 0.04922898778857084, 0.05580114068309453),
    (0.02385199249245906, 0.02093905186688443, 0.09482952367831235),
    (0.06861856936317437, 0.04153859183110701, 0.059716307046232514),
]


@pytest.mark.parametrize("ions", [False, True])
@pytest.mark.parametrize("offset", TIES)
def test_pair_at_the_cutoff(device_lib, oracle_lib, offset, ions):
    pair = np.array([(0.0, 0.0, 0.0), offset])
    far = np.array([(500.0, 0.0, 0.0)])
    x_el, x_ion = (far, pair) if ions else (pair, far)
    n_el, n = len(x_el), 3
    cfg = api.Config(physics=api.PHYS_REF)
    r = oracle.direct(x_el, x_ion, oracle.make_params(
        theta=0.5, rs=units.kelbg_lambdas(cfg.te)[1], physics=api.PHYS_REF))
    g = np.vstack([r["f_el"], r["f_ion"]])
    with api.TreeForce(n_el, n - n_el, cfg) as tf:
        z = [np.zeros_like(a) for a in (x_el, x_el, x_ion, x_ion)]
        tf.load_state(x_el, z[0], z[1], x_ion, z[2], z[3])
        f, e = tf.direct(np.arange(n))
    assert (np.abs(f - g) <= 1e-12 * np.abs(g).max()).all()
    assert e.sum() == pytest.approx(r["epot"], rel=1e-12)
