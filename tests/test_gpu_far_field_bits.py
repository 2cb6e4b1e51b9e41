"""The mixed walk's forces to the last bit.

A loop of steps amplifies a difference in the last bit of a force through the
close passages of the electrons, so the order of the walk's operations is part
of its results: sums, contractions and the order of the batches stay as they
are.  The digests are SHA-256 (first 16 digits) of the forces of a cloud made
by exact operations, one per size of team (16, 8, 4, 2 warps, 1 warp), order of
the far field and build (without and with RDF counts).  They belong to
CUDA 12.9; another compiler may round elsewhere.
"""
import hashlib

import numpy as np
import pytest

from tree_b200 import api, learned_mac

pytestmark = pytest.mark.gpu

SIZES = (1999, 4501, 9001, 20001, 33000)
DIGESTS = {
    (1999, 2, False): ("bad12302a62e3e9d", "3c51f39216ed9501"),
    (1999, 3, False): ("1775301e69b7350f", "6cb7dba6821b138a"),
    (1999, 4, False): ("7bd51890c296caa6", "3811c79de863b000"),
    (1999, 3, True): ("e43d9e199f8f9d8d", "20f194374d0db6aa"),
    (1999, 4, True): ("0afb9f395994849a", "80231a6a88af89a4"),
    (4501, 2, False): ("6e54541033e316b4", "cbef3e9f465a1e62"),
    (4501, 3, False): ("f974df853015bfe0", "98e736d092d0f034"),
    (4501, 4, False): ("7589399ba29dabfe", "8384c93f6d0a3f3f"),
    (4501, 3, True): ("d11ade7fd9eb2236", "5e939d36496c8e68"),
    (4501, 4, True): ("b1666982aa007477", "543c8d10992dca6f"),
    (9001, 2, False): ("402a367650a0c34d", "07dfbb12cc5c8797"),
    (9001, 3, False): ("1bc77f75e6a376be", "01be73a782e200f3"),
    (9001, 4, False): ("78744640c47f28c3", "3b8c64517864ee4f"),
    (9001, 3, True): ("71ce35870612c04a", "89d2fc71c99680f9"),
    (9001, 4, True): ("2e0e180eaa5a03e8", "d0fbeae20bbfbbbc"),
    (20001, 2, False): ("d5482ee1b046f32d", "14460259331dc4dd"),
    (20001, 3, False): ("0ac968a33294f410", "98d0968d7327a3d1"),
    (20001, 4, False): ("9020a64fbfbe64db", "f5a55bf07ec02dea"),
    (20001, 3, True): ("396a66a4fc4d1474", "e8aec0f5b6544c24"),
    (20001, 4, True): ("28793dde5c90ba8a", "4005566094255c47"),
    (33000, 2, False): ("b8baa117bfbce131", "b0439a16d2bdcbca"),
    (33000, 3, False): ("c12f91fc71d6bb81", "027d556ac920198b"),
    (33000, 4, False): ("4b440cc6c12bff46", "cc60ffa133388cd2"),
    (33000, 3, True): ("16ff97b42b01c8f8", "f85cdf5e145f70ad"),
    (33000, 4, True): ("71c5206fe5ddecdf", "6e71eb922b7beda5"),
}


def _cloud(n):
    """Sums of uniform numbers: the same bits with every NumPy and processor."""
    rng = np.random.Generator(np.random.Philox(n))
    n_ion = (n + 1) // 2
    u = rng.random((8, n_ion, 3))
    x_ion = (u[0] + u[1] + u[2] + u[3] - 2.0) * 32.0
    x_el = x_ion + (u[4] + u[5] + u[6] + u[7] - 2.0) * 0.5
    return x_el[:n - n_ion], x_ion


def _digests(n, order, learned):
    x_el, x_ion = _cloud(n)
    cfg = api.Config(theta=0.42, physics=api.PHYS_KELBG, precision=api.PREC_MIXED,
                     mac=api.MAC_LEARNED if learned else api.MAC_FIXED)
    got = []
    with api.TreeForce(len(x_el), len(x_ion), cfg) as tf:
        tf.set_tuning(8, 4, order)
        if learned:
            params, stats, _ = learned_mac.load_model(order=order)
            tf.mac_set_model(params, stats)
            tf.mac_config(3e-5, 0.05, 0.9)
        for rdf in (False, True):
            bins = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)] if rdf else (None, None)
            f = np.vstack(tf.force(x_el, x_ion, *bins)[:2]) + 0.0  # one sign of zero
            got.append(hashlib.sha256(f.tobytes()).hexdigest()[:16])
    return tuple(got)


@pytest.mark.parametrize("order,learned", [(2, False), (3, False), (4, False), (3, True),
                                           (4, True)])
@pytest.mark.parametrize("n", SIZES)
def test_forces_to_the_last_bit(device_lib, n, order, learned):
    assert _digests(n, order, learned) == DIGESTS[n, order, learned]
