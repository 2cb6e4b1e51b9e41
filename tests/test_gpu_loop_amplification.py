"""Ten steps of the mixed path against ten steps with the forces of the FP64
direct sum on every particle.

The electrons' close passages amplify any error of a force, so the positions
after a loop have no bound of their own.  Each particle is held to what errors
of the mixed path's size do to it: loops with the direct sum's forces plus, on
every particle and step, a vector as long as the mixed path's own error there,
in a direction that a particle keeps for the loop (errors of a slowly changing
tree add up).  Where positions answer linearly, such a loop parts from the
exact one by as much as the mixed loop may at most.  On a close passage the
difference depends on the direction, through a cosine: it exceeds KEEP times
the largest of LOOPS with probability KEEP**-LOOPS, 2e-5.  The walk's rounding
(the order in which it adds) is far inside.
"""
import numpy as np
import pytest

from tree_b200 import api, cloud, units

pytestmark = pytest.mark.gpu

N, STEPS, LOOPS, KEEP = 32768, 10, 4, 16.0
DT = units.dt_code(1e-11)
MASS = np.repeat([units.M_ELECTRON_AMU, units.M_ION_AMU], N // 2)[:, None]


def _state():
    c = cloud.make_cloud(N, seed=41, te_k=50.0, n0_per_m3=1e15)
    rng = np.random.Generator(np.random.Philox(42))
    x_el = c.x_ion + c.v_el * (20.0 * DT)  # the electrons left their ions 20 steps ago
    x, v = np.vstack([x_el, c.x_ion]), np.vstack([c.v_el, c.v_ion])
    return x, v, rng


def _loop(tf, x, v, f, change):
    """Velocity Verlet with the direct sum's forces, changed by change(step, x, f)."""
    ne, every = N // 2, np.arange(N)
    x, v, f = x.copy(), v.copy(), f.copy()
    for step in range(STEPS):
        v += 0.5 * DT * f / MASS
        x += DT * v
        tf.load_state(x[:ne], v[:ne], f[:ne], x[ne:], v[ne:], f[ne:])
        f = change(step, x, tf.direct(every)[0])
        v += 0.5 * DT * f / MASS
    return x


def test_ten_mixed_steps_stay_within_their_own_errors(device_lib):
    x0, v0, rng = _state()
    ne = N // 2
    cfg = api.Config(theta=0.42, physics=api.PHYS_KELBG, precision=api.PREC_MIXED)
    with api.TreeForce(ne, ne, cfg) as tf, api.TreeForce(ne, ne, cfg) as mixed:
        mixed.set_tuning(8, 3, 4)
        tf.load_state(x0[:ne], v0[:ne], v0[:ne], x0[ne:], v0[ne:], v0[ne:])
        f0 = tf.direct(np.arange(N))[0]
        mixed.load_state(x0[:ne], v0[:ne], f0[:ne], x0[ne:], v0[ne:], f0[ne:])
        mixed.step(DT, STEPS)
        st = mixed.get_state()
        got = np.vstack([st["x_el"], st["x_ion"]])

        exact = _loop(tf, x0, v0, f0, lambda step, x, f: f)
        bound = np.zeros(N)
        for _ in range(LOOPS):
            way = rng.standard_normal((N, 3))
            way /= np.linalg.norm(way, axis=1, keepdims=True)

            def noisy(step, x, f):
                off = np.vstack(mixed.force(x[:ne], x[ne:])[:2]) - f
                return f + way * np.linalg.norm(off, axis=1, keepdims=True)

            part = np.linalg.norm(_loop(tf, x0, v0, f0, noisy) - exact, axis=1)
            bound = np.maximum(bound, part)
        # a particle whose error happens to vanish: a tenth of its species' median
        for sp in (slice(0, ne), slice(ne, N)):
            bound[sp] = np.maximum(bound[sp], 0.1 * np.median(bound[sp]))

        # the same loop without one near pair's force on an electron, in one step
        victim = int(np.argmin(np.abs(np.linalg.norm(x0[:ne] - x0[ne:], axis=1) - 1.0)))

        def without_a_pair(step, x, f):
            if step == 2:
                d = x[victim] - x[ne:]
                r2 = (d * d).sum(1)
                j = int(np.argmin(r2))
                f = f.copy()
                f[victim] += units.EPS * d[j] / r2[j] ** 1.5
            return f

        lost = _loop(tf, x0, v0, f0, without_a_pair)
    off = np.linalg.norm(got - exact, axis=1)
    assert (off <= KEEP * bound).all(), (off / bound).max()
    assert np.linalg.norm(lost - exact, axis=1)[victim] > KEEP * bound[victim]
