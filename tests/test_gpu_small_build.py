"""The small build (counting sort, one-block passes) and the sort without scans at
their edges: trees equal to the oracle's bit for bit on the FP64 path, and on the
mixed path the sorted particles, cells and moments of every twig."""
import numpy as np
import pytest

import oracle
from tree_b200 import api

pytestmark = pytest.mark.gpu


def _points(n, seed, tight):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, 3)) * 30.0
    if tight and n > 3:
        # a long run of equal high key words, and pairs of them
        x[1:] = rng.standard_normal((n - 1, 3)) * 1e-6
        x[0] = 1e3
        x[n // 2:] = rng.standard_normal((n - n // 2, 3)) * 30.0
    return x


@pytest.mark.parametrize("tight", [False, True])
@pytest.mark.parametrize("n_el,n_ion", [(1, 0), (1, 2), (40, 0), (0, 33), (700, 333), (2100, 2300),
                                        (6143, 6145), (6144, 6145), (8192, 8193)])
def test_fp64_trees(device_lib, oracle_lib, n_el, n_ion, tight):
    x_el, x_ion = _points(n_el, n_el + 1, tight), _points(n_ion, n_ion + 2, tight)
    with api.TreeForce(n_el, n_ion, api.Config(theta=0.7, precision=api.PREC_FP64)) as tf:
        tf.force(x_el, x_ion)
        dumps = [tf.tree_dump(0), tf.tree_dump(1)]
    for dev, x, sign in zip(dumps, (x_el, x_ion), (-1, 1)):
        if len(x) == 0:
            assert len(dev["level"]) == 0
            continue
        ref, _ = oracle.tree_dump(x, sign)
        np.testing.assert_array_equal(dev["level"], ref["level"])
        np.testing.assert_array_equal(dev["skip"], ref["skip"])
        leaf = ref["ileaf"] != 0
        np.testing.assert_array_equal(dev["pt"][leaf], ref["pt"][leaf])
        np.testing.assert_array_equal(dev["centre"], ref["xx"])
        np.testing.assert_array_equal(
            dev["moments"], np.concatenate([ref["qeff"][:, None], ref["D"], ref["Q"], ref["QQ"]], 1))


@pytest.mark.parametrize("tight", [False, True])
@pytest.mark.parametrize("n_el,n_ion", [(1, 1), (40, 33), (1024, 1024), (1024, 1025), (6144, 6144),
                                        (6144, 6145), (131072, 131072), (131073, 131072)])
def test_mixed_tree(device_lib, n_el, n_ion, tight):
    x_el, x_ion = _points(n_el, n_el + 1, tight), _points(n_ion, n_ion + 2, tight)
    cfg = api.Config(theta=0.7, physics=api.PHYS_KELBG, precision=api.PREC_MIXED)
    with api.TreeForce(n_el, n_ion, cfg) as tf:
        tf.force(x_el, x_ion)
        d = tf.net_dump()
    p = d["sorted"]
    x = np.vstack([x_el, x_ion])
    np.testing.assert_array_equal(np.sort(p[:, :3], 0), np.sort(x, 0))
    first, count, parent = d["first"], d["count"], d["parent"]
    assert count[0] == len(x) and parent[0] == -1
    inside = (first >= first[parent]) & (first + count <= first[parent] + count[parent])
    assert inside[1:].all()
    twig = np.bincount(parent[1:], minlength=len(count)) > 0
    np.testing.assert_array_equal(
        np.bincount(parent[1:], weights=count[1:], minlength=len(count))[twig], count[twig])
    for t in np.nonzero(twig)[0][:: max(1, int(twig.sum()) // 300)]:
        q = p[first[t]:first[t] + count[t]]
        X = q[:, :3].mean(0)
        a, s = q[:, :3] - X, np.where(q[:, 3] > 0.5, 1.0, -1.0)
        size = max(np.abs(a).max(), 1e-12 * np.abs(X).max(), 1e-300)
        m = d["moments"][t]
        np.testing.assert_allclose(d["centre"][t], X, rtol=1e-12, atol=1e-12 * size)
        assert m[0] == count[t] and m[1] == s.sum()
        assert np.abs(m[2:5] - (s[:, None] * a).sum(0)).max() <= 1e-11 * count[t] * size + 1e-12 * np.abs(X).max() * count[t]
        xxxx = (s * a[:, 0] ** 4).sum()
        assert abs(m[22] - xxxx) <= 1e-10 * count[t] * size ** 4 + 1e-40
