"""The FP64 direct sum at the edges of its tiles and laws against the oracle
(1e-12, the direct-sum bar), several calls on one handle with one scratch."""
import numpy as np
import pytest

import oracle
from tree_b200 import api, units

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics", [api.PHYS_REF, api.PHYS_KELBG])
@pytest.mark.parametrize("n_el,n_ion,scale", [
    (1, 1, 1.0),
    (127, 2, 1.0),       # the species change one source before a tile's end
    (128, 128, 0.01),    # on a tile's end; pairs inside the Kelbg cores
    (0, 130, 1.0),
    (1300, 1111, 30.0),  # several source chunks
])
def test_direct_tiles_and_laws(device_lib, oracle_lib, n_el, n_ion, scale, physics):
    n = n_el + n_ion
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 3)) * scale
    cfg = api.Config(rs=0.5, physics=physics)
    lam = units.kelbg_lambdas(cfg.te)
    p = oracle.make_params(theta=0.5, rs=0.5, lambdas=lam, physics=physics)
    r = oracle.direct(x[:n_el], x[n_el:], p, np.arange(n_el), np.arange(n_ion))
    g = np.vstack([r["f_el"], r["f_ion"]])
    v = np.zeros_like(x)
    with api.TreeForce(n_el, n_ion, cfg) as tf:
        tf.load_state(x[:n_el], v[:n_el], v[:n_el], x[n_el:], v[n_el:], v[n_el:])
        for t in (np.arange(1), np.arange(n), rng.permutation(n)[:(n + 1) // 2]):
            f, e = tf.direct(t)
            nrm = np.linalg.norm(g[t], axis=1)
            assert (np.linalg.norm(f - g[t], axis=1)
                    <= 1e-12 * np.maximum(nrm, 1e-3 * np.linalg.norm(g, axis=1).max())).all()
            if len(t) == n:
                assert e.sum() == pytest.approx(r["epot"], rel=1e-12)
