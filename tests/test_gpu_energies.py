"""Potential energies, electrons' and ions' shares apart, at the edges of the
walks' layouts and batches.

FP64 walk: against the oracle, within 1e-12 of the gross sum eps/2 sum 1/r (a
particle's sum has some thousand terms, regrouped: 1e3 roundings of 1.1e-16).
Mixed walk with every cell opened: against the FP64 walk, within 4e-6 of the
gross sum (a pair's FP32 distance is within 7.3e-7 of the exact one, its inverse
root within 2.4e-7, and 16 terms are added in FP32).
"""
import numpy as np
import pytest
import torch

import oracle
from tree_b200 import api, cloud, units

pytestmark = pytest.mark.gpu


def _gross(x):
    xt = torch.from_numpy(x).cuda()
    s = 0.0
    for k in range(0, len(x), 2048):
        r = torch.cdist(xt[k:k + 2048], xt, compute_mode="donot_use_mm_for_euclid_dist")
        s += float(torch.where(r > 0, 1.0 / r, 0.0).sum())
    return 0.5 * units.EPS * s


@pytest.mark.parametrize("physics", [api.PHYS_REF, api.PHYS_KELBG])
@pytest.mark.parametrize("n_el,n_ion,scale,rs", [
    (1, 1, 1.0, None),
    (33, 5, 1.0, 0.5),         # pairs inside the screening length
    (6143, 6144, 60.0, None),  # the last size with a warp per target
    (6145, 6144, 60.0, None),  # four targets a warp, a short last group
    (0, 12291, 60.0, None),
    (40, 37, 1e38, 1e30),      # the plain divisions
])
def test_fp64_walk(device_lib, oracle_lib, n_el, n_ion, scale, rs, physics):
    x = np.random.default_rng(n_el + n_ion).standard_normal((n_el + n_ion, 3)) * scale
    cfg = api.Config(theta=0.6, rs=rs, physics=physics, precision=api.PREC_FP64)
    lam = units.kelbg_lambdas(cfg.te)
    r = oracle.force(x[:n_el], x[n_el:], oracle.make_params(theta=0.6, rs=rs or lam[1],
                                                            lambdas=lam, physics=physics))
    with api.TreeForce(n_el, n_ion, cfg) as tf:
        _, _, ee, ei = tf.force(x[:n_el], x[n_el:])
    tol = 1e-12 * _gross(x)
    assert abs(ee - r["epot_e"]) <= tol and abs(ei - r["epot_i"]) <= tol


@pytest.mark.parametrize("physics", [api.PHYS_REF, api.PHYS_KELBG])
@pytest.mark.parametrize("n_el,n_ion", [
    (1, 1), (17, 16), (31, 32), (0, 33), (40, 0),            # ends of a batch of sources
    (700, 699), (2100, 2101), (5000, 5001), (9000, 9000), (15000, 15001),  # teams 16, 8, 4, 2, 1
])
def test_mixed_walk_of_every_pair(device_lib, n_el, n_ion, physics):
    c = cloud.make_cloud(2 * max(n_el, n_ion), seed=n_el + 5)
    rng = np.random.default_rng(n_ion)
    x = np.vstack([c.x_ion[:n_el] + rng.standard_normal((n_el, 3)) * 0.3, c.x_ion[:n_ion]])
    got = {}
    for prec in (api.PREC_FP64, api.PREC_MIXED):
        cfg = api.Config(theta=1e-9, physics=physics, precision=prec)
        with api.TreeForce(n_el, n_ion, cfg) as tf:
            got[prec] = tf.force(x[:n_el], x[n_el:])[2:]
    tol = 4e-6 * _gross(x)
    for a, b in zip(got[api.PREC_MIXED], got[api.PREC_FP64]):
        assert abs(a - b) <= tol


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("local", [0.0, 0.08])
@pytest.mark.parametrize("n", [4000, 32000])  # a team, one warp
def test_far_field_split(device_lib, n, local, order):
    # A far cell's ions enter the ions' energy as one charge at the centroid of
    # all its particles.  Its half-diagonal is below sqrt(3)/2 theta d, so at
    # theta = 0.2 the share is within 0.173 / (1 - 0.173) = 0.21 of itself; the sum
    # of both energies has the whole expansion (rms 1e-4 of the gross sum).
    h = n // 2
    c = cloud.make_cloud(n, seed=n)
    x_el = c.x_ion + np.random.default_rng(n).standard_normal((h, 3)) * 0.3
    x = np.vstack([x_el, c.x_ion])
    cfg = api.Config(theta=1e-9, physics=api.PHYS_KELBG, precision=api.PREC_FP64)
    with api.TreeForce(h, h, cfg) as tf:
        _, _, ee64, ei64 = tf.force(x_el, c.x_ion)
    cfg = api.Config(theta=0.2, physics=api.PHYS_KELBG, precision=api.PREC_MIXED)
    for rdf in (False, True):
        bins = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)] if rdf else (None, None)
        with api.TreeForce(h, h, cfg) as tf:
            tf.set_tuning(8, 4, order)
            tf.set_local_expansion(local)
            _, _, ee, ei = tf.force(x_el, c.x_ion, *bins)
            t = tf.timings()
        assert t.n_m2p > 0 and (t.n_local > 0) == (local > 0)
        assert abs(ei - ei64) <= 0.21 * _gross(c.x_ion)
        assert abs(ee + ei - ee64 - ei64) <= 1e-4 * _gross(x)
