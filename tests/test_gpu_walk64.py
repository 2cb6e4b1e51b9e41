"""The FP64 walk at the edges of its two layouts (one and four targets per
warp) against the oracle: the same decisions and counts, forces to 1e-10."""
import numpy as np
import pytest

import oracle
from tree_b200 import api, units

pytestmark = pytest.mark.gpu


def _compare(x_el, x_ion, theta, physics, rs):
    cfg = api.Config(theta=theta, rs=rs, physics=physics, precision=api.PREC_FP64)
    rdf = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)]
    with api.TreeForce(len(x_el), len(x_ion), cfg) as tf:
        f_el, f_ion, ee, ei = tf.force(x_el, x_ion, *rdf)
        t = tf.timings()
    lam = units.kelbg_lambdas(cfg.te)
    r = oracle.force(x_el, x_ion, oracle.make_params(theta=theta, rs=rs or lam[1], dx_ei=0.01,
                                                     dx_ii=0.1, lambdas=lam, physics=physics))
    f, g = np.vstack([f_el, f_ion]), np.vstack([r["f_el"], r["f_ion"]])
    nrm = np.linalg.norm(g, axis=1)
    assert (np.linalg.norm(f - g, axis=1) <= 1e-10 * np.maximum(nrm, 1e-3 * nrm.max())).all()
    assert (t.n_m2p, t.n_p2p) == (r["stats"]["n_m2p"], r["stats"]["n_p2p"])
    np.testing.assert_array_equal(rdf[0], r["rdf_ei"])
    np.testing.assert_array_equal(rdf[1], r["rdf_ii"])


@pytest.mark.parametrize("physics", [api.PHYS_REF, api.PHYS_KELBG])
@pytest.mark.parametrize("n_el,n_ion,scale,rs", [
    (6143, 6144, 60.0, None),    # the last size with a warp per target
    (6145, 6144, 60.0, None),    # shared walks: a group across the species, a short last group
    (0, 12291, 60.0, None),      # one tree, shared
    (33, 5, 1.0, 0.5),           # pairs inside the screening length
    (40, 37, 1e38, 1e30),        # seventh powers near the end of the exponent range
])
def test_layout_edges(device_lib, oracle_lib, n_el, n_ion, scale, rs, physics):
    rng = np.random.default_rng(n_el + n_ion)
    x = rng.standard_normal((n_el + n_ion, 3)) * scale
    _compare(x[:n_el], x[n_el:], 0.6, physics, rs)


def test_colocated_noise_in_a_shared_walk(device_lib, oracle_lib):
    # every electron on its ion: forces cancel to rounding noise, which only
    # the reference's own order of operations reproduces
    x = np.random.default_rng(3).standard_normal((6200, 3)) * 60.0
    _compare(x, x.copy(), 0.6, api.PHYS_REF, None)


@pytest.mark.parametrize("side,theta", [(12, 0.5), (24, 0.5), (24, 1.0)])
def test_ties_of_the_acceptance_test(device_lib, oracle_lib, side, theta):
    # lattice points at powers of two: many cells lie exactly at the limit, or
    # within rounding of it, where the squared test falls back to the root
    g = (np.arange(side) - side // 2).astype(float)
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) * 4.0
    x[:] = x[np.random.default_rng(side).permutation(len(x))]
    _compare(x[::2], x[1::2], theta, api.PHYS_REF, None)
