"""The mixed walk's direct pairs (theta -> 0: every cell opened) at the edges of
its batches: forces against the FP64 direct sum, RDF bins against FP64
distances.  A pair within 3e-6 of a bin edge (FP32 distance) may fall in the
neighbouring bin; the totals are exact."""
import numpy as np
import pytest

from tree_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics", [api.PHYS_REF, api.PHYS_KELBG])
@pytest.mark.parametrize("n_el,n_ion,scale,rs", [
    (1, 1, 1.0, None),
    (17, 16, 1.0, None),     # one source past a batch
    (0, 33, 1.0, None),
    (40, 0, 1.0, None),
    (31, 32, 0.01, None),    # pairs inside the Kelbg cores and the cutoff
    (70, 77, 2.0, 0.8),      # most e-i pairs inside the screening length
    (300, 211, 40.0, None),  # pairs beyond the last e-i bin
])
def test_pairs_and_rdf_bins(device_lib, n_el, n_ion, scale, rs, physics):
    rng = np.random.default_rng(n_el + 7 * n_ion)
    x = rng.standard_normal((n_el + n_ion, 3)) * scale
    ion = np.arange(n_el + n_ion) >= n_el
    cfg = api.Config(theta=1e-9, rs=rs, physics=physics, precision=api.PREC_MIXED, dx_ei=0.004,
                     dx_ii=0.03)
    rdf = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)]
    with api.TreeForce(n_el, n_ion, cfg) as tf:
        f_el, f_ion, _, _ = tf.force(x[:n_el], x[n_el:], *rdf)
        fd, _ = tf.direct(np.arange(len(x)))
    f = np.vstack([f_el, f_ion])
    # a pair is within a few FP32 roundings of its law; the e-i screening law
    # subtracts terms (rs/r)^2 larger than itself
    r2 = ((x[:, None] - x[None]) ** 2).sum(-1)
    gross = 0.00144 * (1.0 / np.maximum(r2 + np.eye(len(x)) * 1e30, 1e-30)).sum(1)
    if rs is not None or physics == api.PHYS_KELBG:
        gross = np.maximum(gross, np.linalg.norm(fd, axis=1))
    assert (np.linalg.norm(f - fd, axis=1) <= 4e-6 * gross + 1e-30).all()
    r = np.sqrt(r2)
    same = ion[:, None] == ion[None]
    off = ~np.eye(len(x), dtype=bool)
    counted = [off & ~same, off & same & ion[:, None]]
    if physics == api.PHYS_REF:
        counted[1] &= r2 > 0.01
    for got, mask, dx in zip(rdf, counted, (0.004, 0.03)):
        t = r[mask] / dx
        sure = np.abs(t - np.round(t)) > 3e-6 * np.maximum(t, 1.0)
        lo = np.bincount(np.minimum(t[sure], api.RDF_BINS).astype(int), minlength=api.RDF_BINS + 1)
        hi = lo.copy()
        for v in t[~sure]:  # either side of the edge
            for b in (int(np.round(v)) - 1, int(np.round(v))):
                hi[min(max(b, 0), api.RDF_BINS)] += 1
        assert (got >= lo[:-1]).all() and (got <= hi[:-1]).all()
        inside = int((t[sure] < api.RDF_BINS).sum())
        assert inside <= got.sum() <= inside + int((~sure).sum())
