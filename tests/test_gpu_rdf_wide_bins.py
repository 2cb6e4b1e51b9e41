"""RDF bins of any width count pairs of particles only: the empty places of a
batch of sources, which the walk fills with chargeless dummies, fall in none."""
import numpy as np
import pytest

from tree_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics", [api.PHYS_REF, api.PHYS_KELBG])
@pytest.mark.parametrize("width", [1e3, 1e15, 1e17, 1e30])
@pytest.mark.parametrize("n_el,n_ion", [(16, 17), (1, 2), (2000, 1999)])
def test_all_pairs_in_the_first_bin(device_lib, n_el, n_ion, width, physics):
    rng = np.random.default_rng(n_el)
    x = rng.standard_normal((n_el + n_ion, 3)) * 30.0
    cfg = api.Config(theta=1e-9, physics=physics, precision=api.PREC_MIXED, dx_ei=width,
                     dx_ii=width)
    rdf = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)]
    with api.TreeForce(n_el, n_ion, cfg) as tf:
        tf.force(x[:n_el], x[n_el:], *rdf)
    r2 = ((x[n_el:, None] - x[None, n_el:]) ** 2).sum(-1)
    ii = n_ion * (n_ion - 1) if physics == api.PHYS_KELBG else int((r2 > 0.01).sum())
    assert (rdf[0][0], rdf[1][0]) == (2 * n_el * n_ion, ii)
    assert rdf[0][1:].sum() == 0 and rdf[1][1:].sum() == 0
