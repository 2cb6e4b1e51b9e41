"""Small clouds, whose target groups are shared by teams of warps: at the sizes
where the team changes, every pair is summed exactly once, results repeat bit
for bit and equal those of the same cloud inside a large ensemble (one warp per
group), and accuracy is the mixed path's."""
import numpy as np
import pytest

from tree_b200 import api, cloud, learned_mac, units

pytestmark = pytest.mark.gpu


def _plasma(n_el, n_ion):
    c = cloud.make_cloud(2 * max(n_el, n_ion), seed=n_el + 5)
    rng = np.random.Generator(np.random.Philox(n_ion))
    return c.x_ion[:n_el] + rng.standard_normal((n_el, 3)) * 0.3, c.x_ion[:n_ion]


@pytest.mark.parametrize("n_el,n_ion", [(1, 0), (1, 1), (16, 17), (1499, 1500), (1500, 1500),
                                        (2999, 3000), (3000, 3001), (9999, 10000),
                                        (10000, 10000)])
def test_every_pair_once(device_lib, n_el, n_ion):
    x_el, x_ion = _plasma(n_el, n_ion)
    n = n_el + n_ion
    cfg = api.Config(theta=1e-9, physics=api.PHYS_KELBG, precision=api.PREC_MIXED, dx_ei=1.0,
                     dx_ii=1.0)
    for rdf in (False, True):
        bins = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)] if rdf else (None, None)
        with api.TreeForce(n_el, n_ion, cfg) as tf:
            f_el, f_ion, _, _ = tf.force(x_el, x_ion, *bins)
            t = tf.timings()
            fd, _ = tf.direct(np.arange(n))
        assert (t.n_m2p, t.n_local, t.n_p2p) == (0, 0, n * n)
        if rdf:
            assert bins[0].sum() == 2 * n_el * n_ion and bins[1].sum() == n_ion * (n_ion - 1)
        err = np.linalg.norm(np.vstack([f_el, f_ion]) - fd, axis=1)
        nrm = np.linalg.norm(fd, axis=1)
        assert np.sqrt(np.mean((err / np.maximum(nrm, 1e-30)) ** 2)) < 4e-6 or n < 3


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("n", [100, 600, 2998, 3000, 5998, 6000, 19998, 20000])
def test_accuracy_and_repeatability(device_lib, n, learned):
    x_el, x_ion = _plasma(n // 2, n // 2)
    v = np.zeros_like(x_el)
    cfg = api.Config(theta=0.42, physics=api.PHYS_KELBG, precision=api.PREC_MIXED,
                     mac=api.MAC_LEARNED if learned else api.MAC_FIXED)
    with api.TreeForce(n // 2, n // 2, cfg) as tf:
        tf.set_tuning(8, 4, 4)
        params, stats, _ = learned_mac.load_model(order=4)
        tf.mac_set_model(params, stats)
        tf.mac_config(3e-5, 0.05, 0.9)
        got = []
        for _ in range(2):
            tf.set_state(x_el, v, x_ion, v)
            _, rdf = tf.run(units.dt_code(1e-13), 2, rdf=True)
            st, t = tf.get_state(), tf.timings()
            got.append((st["f_el"], st["f_ion"], *rdf, np.array([t.n_m2p, t.n_p2p, t.n_local,
                                                                 t.n_mac_net])))
        targets = np.sort(np.random.default_rng(1).choice(n, min(n, 2048), replace=False))
        fd, _ = tf.direct(targets)
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    assert not learned or n < 3000 or got[0][4][3] > 0
    f = np.vstack(got[0][:2])[targets]
    err = np.linalg.norm(f - fd, axis=1) / np.linalg.norm(fd, axis=1)
    assert np.sqrt(np.mean(err**2)) < 1e-4


@pytest.mark.parametrize("learned", [False, True])
def test_a_team_gives_one_warps_bits(device_lib, learned):
    sizes = [(60, 61), (700, 699), (2100, 2100), (8000, 8000), (20000, 20000)]
    cl = [_plasma(*s) for s in sizes]
    cfg = api.Config(theta=0.42, physics=api.PHYS_KELBG, precision=api.PREC_MIXED,
                     mac=api.MAC_LEARNED if learned else api.MAC_FIXED)
    model = learned_mac.load_model(order=4)[:2]

    def tuned(tf):
        tf.set_tuning(8, 4, 4)
        tf.mac_set_model(*model)
        tf.mac_config(3e-5, 0.05, 0.9)
        return tf

    x = np.vstack([np.vstack(c) for c in cl])
    with tuned(api.Ensemble([cfg] * len(cl), [s[0] for s in sizes], [s[1] for s in sizes])) as ens:
        ens.set_state(x, np.zeros_like(x))
        ens.step(units.dt_code(1e-13), 1)
        fe = ens.get_state()["f"]
        for k, (c, s) in enumerate(zip(cl, sizes)):
            with tuned(api.TreeForce(*s, cfg)) as tf:
                tf.set_state(c[0], np.zeros_like(c[0]), c[1], np.zeros_like(c[1]))
                tf.step(units.dt_code(1e-13), 1)
                st = tf.get_state()
            np.testing.assert_array_equal(fe[ens.offsets[k]:ens.offsets[k + 1]],
                                          np.vstack([st["f_el"], st["f_ion"]]))


@pytest.mark.parametrize("n", [15998, 16000, 29998, 30000])
def test_teams_of_two(device_lib, n):
    test_every_pair_once(device_lib, n // 2, n // 2)
    for learned in (False, True):
        test_accuracy_and_repeatability(device_lib, n, learned)
