"""The work that users of the force path have it do, as measurable cases.

A case names an entry point (`call`), a cloud (`n_el` electrons, `n_ion` ions,
peak density 1e15 m^-3, electron temperature `te`) and the method's settings:

  force     TreeForce.force: the drop-in for the reference's CALL Force, host
            arrays in and out, with or without the pair-distance histograms
  step      TreeForce.load_state + run(1 step) + get_state through page-locked
            buffers: a host program that keeps the particle state itself
  loop      TreeForce.load_state + step(dt, steps) + get_state: the
            device-resident step loop between two snapshots
  ensemble  the step of many independent clouds in one handle, of n_el to
            n_ion particles each
  direct    TreeForce.direct: the FP64 direct sum over listed targets, the
            accuracy audit that goes with a run

The clouds are Gaussian clouds of ions with their electrons some time after
ionisation: every electron has moved away from the ion it started on with its
thermal velocity, a few in a thousand were ejected much faster and stretch the
root box, which is what trees meet a few tens of steps into a run.  The forces
that `load_state` takes beside positions and velocities are the pull of that
ion.  Results of the FP32 walk, which the C interface hands out in arrays of
doubles, are kept as the float32 numbers they are; results of the FP64 path
and positions that no FP32 sum went into stay float64.
"""
import math
import random

import numpy as np
import torch

from tree_b200 import api, cloud, learned_mac, units

DT = units.dt_code(1e-11)
SEED_STRIDE = 7919

# defaults of a case's settings
BASE = dict(call="force", n_el=2048, n_ion=2048, te=50.0, precision="mixed", laws="kelbg",
            mac="fixed", theta=0.5, order=3, eta=0.0, rdf=False, steps=1, clouds=1, targets=0)


def _case(name, **kw):
    c = dict(BASE)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one Force call of the plain method at the smallest published size
        _case("force_fp64_4k", precision="fp64", laws="ref", rdf=True),
        # the plain method at its production size
        _case("force_fp64_256k", n_el=131072, n_ion=131072, precision="fp64", laws="ref", rdf=True),
        # FP64 steps with the erf-Kelbg laws at a smaller opening angle, as runs
        # that check the mixed path's drift do; a cloud that has lost electrons
        _case("loop_fp64_30k", call="loop", n_el=14999, n_ion=15362, precision="fp64", theta=0.35,
              steps=2),
        # one mixed-precision Force call with the default tuning: latency counts
        _case("force_mixed_4k", rdf=True),
        # a short loop of a tiny cloud: the per-step launches count
        _case("loop_mixed_1k", call="loop", n_el=500, n_ion=501, steps=20),
        # the loop of a mid-size cloud, fixed test, hexadecapole
        _case("loop_mixed_32k", call="loop", n_el=16384, n_ion=16384, theta=0.42, order=4, steps=10),
        # one step with the learned criterion and histograms, odd counts
        _case("step_learned_256k", call="step", n_el=131073, n_ion=131072, mac="learned",
              theta=0.42, eta=3e-5, order=4, rdf=True),
        # the headline: N = 1M, learned criterion, histograms every step
        _case("step_learned_1m", call="step", n_el=524288, n_ion=524288, mac="learned", theta=0.42,
              eta=3e-5, order=4, rdf=True),
        # N = 1M, fixed test, hot electrons, no histograms (the precision form)
        _case("force_mixed_1m", n_el=524288, n_ion=524288, te=200.0, order=4),
        # the largest published single cloud
        _case("step_learned_4m", call="step", n_el=2097152, n_ion=2097152, mac="learned",
              theta=0.42, eta=3e-5, order=4),
        # 64 clouds of 8k-131k particles in one handle
        _case("ensemble_64", call="ensemble", clouds=64, n_el=8192, n_ion=131072, mac="learned",
              theta=0.36, eta=3e-5, order=4),
        # an accuracy audit: 16,384 targets against every particle in FP64
        _case("direct_16k_of_256k", call="direct", n_el=131072, n_ion=131072, targets=16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["force64", "loop64", "force", "force", "loop", "loop", "step", "step",
                       "ensemble", "direct"])
    te = round(rng.uniform(10.0, 200.0), 1)
    laws = rng.choice(["kelbg", "kelbg", "ref"])

    def species(n):  # up to 3 % of the electrons are gone; counts of either parity
        ions = max(2, n // 2 + rng.randint(0, 1))
        return dict(n_el=max(2, int(ions * (1.0 - 0.03 * rng.random()))), n_ion=ions)

    if kind == "force64":
        return _case("", te=te, laws=laws, precision="fp64", theta=round(rng.uniform(0.4, 0.8), 2),
                     rdf=rng.random() < 0.5, **species(_log_int(rng, 1000, 200000)))
    if kind == "loop64":
        return _case("", call="loop", te=te, laws=laws, precision="fp64", steps=2,
                     theta=round(rng.uniform(0.35, 0.7), 2), **species(_log_int(rng, 1000, 60000)))
    if kind == "direct":
        return _case("", call="direct", te=te, laws=laws, targets=_log_int(rng, 256, 16384),
                     **species(_log_int(rng, 2000, 260000)))
    order = rng.choice([2, 3, 4, 4])
    theta = round(rng.uniform(0.3, 0.7) if order == 4 else rng.uniform(0.35, 0.7), 2)
    if kind == "force":
        return _case("", te=te, laws=laws, theta=theta, order=order, rdf=rng.random() < 0.5,
                     **species(_log_int(rng, 1000, 1000000)))
    if kind == "loop":
        n = _log_int(rng, 800, 100000)
        return _case("", call="loop", te=te, laws=laws, theta=theta, order=order,
                     steps=rng.randint(3, 12), **species(n))
    # the learned criterion has models for the octupole and the hexadecapole
    order = rng.choice([3, 4, 4])
    mac = rng.choice(["learned", "learned", "fixed"])
    theta = round(rng.uniform(0.38, 0.5) if order == 4 else rng.uniform(0.28, 0.36), 2)
    lm = dict(mac=mac, eta=3e-5 if mac == "learned" else 0.0)
    if kind == "step":
        return _case("", call="step", te=te, theta=theta, order=order, rdf=rng.random() < 0.6, **lm,
                     **species(_log_int(rng, 2000, 1500000)))
    lo = _log_int(rng, 1000, 8192)
    return _case("", call="ensemble", clouds=rng.randint(2, 40), theta=theta, order=order, n_el=lo,
                 n_ion=lo * rng.randint(2, 10), te=te, **lm)


# ------------------------------------------------------------------ inputs ----
def _plasma(n_el, n_ion, te, seed, n0=1e15):
    """Positions, velocities and previous forces (el, ion) of a cloud whose
    electrons left their ions 20 steps ago."""
    c = cloud.make_cloud(2 * max(n_el, n_ion), seed=seed, te_k=te, n0_per_m3=n0)
    rng = np.random.Generator(np.random.Philox(seed + 1))
    x_ion, v_ion = c.x_ion[:n_ion].copy(), c.v_ion[:n_ion].copy()
    v_el = c.v_el[:n_el].copy()
    fast = rng.random(n_el) < 0.003  # ejected by a close pass of an ion
    v_el[fast] *= np.exp(rng.uniform(0.0, np.log(30.0), (int(fast.sum()), 1)))
    away = v_el * (20.0 * DT)
    x_el = c.x_ion[:n_el] + away
    r2 = (away * away).sum(1, keepdims=True)
    lam = units.kelbg_lambdas(te)[1]
    f_el = -units.EPS * away * (-np.expm1(-r2 / lam**2)) / (r2 * np.sqrt(r2))
    f_ion = np.zeros_like(x_ion)
    m = min(n_el, n_ion)
    f_ion[:m] = -f_el[:m]
    f_ion[m:] = f_el.mean(0)
    return x_el, v_el, f_el, x_ion, v_ion, f_ion


def _clouds(case, seed):
    """Per cloud of an ensemble: (te, n0, its _plasma arrays); sizes and
    densities log-uniform, temperatures uniform, the same for every seed."""
    rng = np.random.default_rng(5)
    k = case["clouds"]
    n = np.exp(rng.uniform(np.log(case["n_el"]), np.log(case["n_ion"]), k)).astype(int)
    n0 = np.exp(rng.uniform(np.log(1e14), np.log(1e16), k))
    te = rng.uniform(10.0, 200.0, k)
    return [(float(te[i]), _plasma(int(n[i]) // 2, (int(n[i]) + 1) // 2, float(te[i]),
                                   seed * 1000 + i, float(n0[i]))) for i in range(k)]


def _config(case, te=None):
    return api.Config(
        theta=case["theta"], te=case["te"] if te is None else te,
        physics=api.PHYS_KELBG if case["laws"] == "kelbg" else api.PHYS_REF,
        precision=api.PREC_FP64 if case["precision"] == "fp64" else api.PREC_MIXED,
        mac=api.MAC_LEARNED if case["mac"] == "learned" else api.MAC_FIXED)


def _tune(tf, case):
    if case["precision"] == "mixed" and (case["order"] != 3 or case["mac"] == "learned"):
        tf.set_tuning(8, 2 if case["mac"] == "learned" else 3, case["order"])
    if case["mac"] == "learned":
        params, stats, _ = learned_mac.load_model(order=case["order"])
        tf.mac_set_model(params, stats)
        tf.mac_config(case["eta"], 0.05, 0.9)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


class _State:
    pass


def prepare(case, seed):
    seed = int(seed) * SEED_STRIDE % (1 << 31)
    s = _State()
    s.case = case
    if case["call"] == "ensemble":
        cl = _clouds(case, seed)
        packed = [np.vstack([np.vstack([c[k], c[k + 3]]) for _, c in cl]) for k in range(3)]
        s.host = [_pinned(a) for a in packed]
        s.back = [torch.empty_like(t).pin_memory() for t in s.host]
        s.tf = api.Ensemble([_config(case, te) for te, _ in cl], [len(c[0]) for _, c in cl],
                            [len(c[3]) for _, c in cl])
        _tune(s.tf, case)
        s.v32, s.f32 = (torch.empty(t.shape, dtype=torch.float32) for t in s.back[1:])
        return s
    x_el, v_el, f_el, x_ion, v_ion, f_ion = _plasma(case["n_el"], case["n_ion"], case["te"], seed)
    s.tf = api.TreeForce(case["n_el"], case["n_ion"], _config(case))
    _tune(s.tf, case)
    if case["call"] == "force":
        s.x_el, s.x_ion = x_el, x_ion
    elif case["call"] == "direct":
        s.tf.load_state(x_el, v_el, f_el, x_ion, v_ion, f_ion)
        rng = np.random.default_rng(seed)
        n = case["n_el"] + case["n_ion"]
        s.targets = np.sort(rng.choice(n, min(case["targets"], n), replace=False))
    else:
        s.host = [_pinned(a) for a in (x_el, v_el, f_el, x_ion, v_ion, f_ion)]
        s.back = [torch.empty_like(t).pin_memory() for t in s.host]
        s.out32 = [torch.empty(t.shape, dtype=torch.float32) for t in s.back]
    return s


# --------------------------------------------------------------------- run ----
def _sums(case, *values):
    """Energies and kinetic sums: double on the FP64 path, the FP32 walk's
    precision on the mixed one."""
    return np.array(values, np.float64 if case["precision"] == "fp64" else np.float32)


def run(s):
    case, tf = s.case, s.tf
    fp64 = case["precision"] == "fp64"
    if case["call"] == "direct":
        f, e = tf.direct(s.targets)
        return {"f": f, "epot": e}
    if case["call"] == "force":
        rdf = [np.zeros(api.RDF_BINS, np.int64) for _ in range(2)] if case["rdf"] else (None, None)
        f_el, f_ion, ee, ei = tf.force(s.x_el, s.x_ion, *rdf)
        out = {"f_el": f_el if fp64 else f_el.astype(np.float32),
               "f_ion": f_ion if fp64 else f_ion.astype(np.float32), "epot": _sums(case, ee, ei)}
        if case["rdf"]:
            out["rdf_ei"], out["rdf_ii"] = rdf
        return out
    if case["call"] == "ensemble":
        x, v, f = (t.data_ptr() for t in s.host)
        tf.load_state(x, v, f)
        tf.step(DT, case["steps"])
        tf.get_state_ptr(*(t.data_ptr() for t in s.back))
        s.v32.copy_(s.back[1])
        s.f32.copy_(s.back[2])
        return {"x": s.back[0], "v": s.v32, "f": s.f32, "sums": tf.sums().astype(np.float32)}
    tf.load_state(*(t.data_ptr() for t in s.host))
    out = {}
    if case["call"] == "step":
        if case["rdf"]:
            rec, (out["rdf_ei"], out["rdf_ii"]) = tf.run(DT, 1, nsamp=1, rdf=True)
        else:
            rec = tf.run(DT, 1, nsamp=1)
        r = rec[0]
        out["sums"] = _sums(case, r["epot_e"], r["epot_i"], r["mv2_el"], r["mv2_ion"],
                            r["rad_el"], r["rad_ion"])
    else:
        d = tf.step(DT, case["steps"])
        out["sums"] = _sums(case, d.epot_e, d.epot_i, d.mv2_el, d.mv2_ion, d.rad_el, d.rad_ion)
    tf.get_state_ptr(*(t.data_ptr() for t in s.back))
    names = ("x_el", "v_el", "f_el", "x_ion", "v_ion", "f_ion")
    for name, t, t32 in zip(names, s.back, s.out32):
        # the first step's positions come from the given forces alone
        if fp64 or (name[0] == "x" and case["steps"] == 1):
            out[name] = t
        else:
            out[name] = t32.copy_(t)
    return out


# -------------------------------------------------------------------- work ----
def work(case):
    """Bytes: the particle data of the call, read and written once.  Flops: the
    method's interactions, about as many per particle as a tree of this size
    and opening angle has (far cells and near pairs, ~ log8(n) / theta^3 of
    each, 50 to 195 flop a far cell by order, 24 to 30 a pair)."""
    def flops(n):
        if case["call"] == "direct":
            return 30.0 * n * min(case["targets"], n)
        far = {2: 50, 3: 100, 4: 195}[case["order"]] if case["precision"] == "mixed" else 194
        lists = min(n, 12.0 * max(1.0, math.log(n, 8)) / case["theta"] ** 3)
        return n * lists * (far + 27)

    if case["call"] == "ensemble":
        rng = np.random.default_rng(5)
        sizes = np.exp(rng.uniform(np.log(case["n_el"]), np.log(case["n_ion"]),
                                   case["clouds"])).astype(int)
    else:
        sizes = [case["n_el"] + case["n_ion"]]
    n = float(sum(sizes))
    per = {"force": 48.0, "direct": 24.0}.get(case["call"], 144.0)
    total = per * n + (32.0 * case["targets"] if case["call"] == "direct" else 0.0)
    if case["rdf"]:
        total += 2 * 8 * api.RDF_BINS
    return {"bytes": total, "flops": case["steps"] * sum(flops(float(k)) for k in sizes)}


# ------------------------------------------------------------------- exact ----
def _exact_forces(case, te, x_el, x_ion, at=None):
    """The direct sum in 64 bits: forces (targets, 3) and 0.5 * sum of V per
    target, split by source (electrons, ions)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cfg = _config(case, te).to_c()
    lam_ee, lam_ei, lam_ii = units.kelbg_lambdas(te)
    x = torch.from_numpy(np.vstack([x_el, x_ion])).to(dev)
    ne, n = len(x_el), len(x_el) + len(x_ion)
    at = torch.arange(n, device=dev) if at is None else torch.from_numpy(at).to(dev)
    force = torch.zeros(len(at), 3, dtype=torch.float64, device=dev)
    pot = torch.zeros(len(at), 2, dtype=torch.float64, device=dev)
    rows = max(1, 48_000_000 // max(1, n))
    for sp, (lo, hi) in enumerate(((0, ne), (ne, n))):
        src = x[lo:hi]
        for tsp in (0, 1):
            idx = torch.nonzero((at >= ne) == bool(tsp)).flatten()
            same = sp == tsp
            lam = lam_ei if not same else (lam_ii if tsp else lam_ee)
            sign = units.EPS if same else -units.EPS
            for k in range(0, len(idx), rows):
                part = idx[k:k + rows]
                xt = x[at[part]]
                d = [xt[:, None, j] - src[None, :, j] for j in range(3)]
                r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
                if case["laws"] == "kelbg":
                    off = r2 == 0.0  # the target itself
                    r = torch.where(off, 1.0, r2).sqrt()
                    g = -torch.expm1(-(r / lam) ** 2)
                    near = r / lam < 6.4
                    v = g / r
                    if bool(near.any()):
                        v = v + math.sqrt(math.pi) / lam * torch.special.erfc(r / lam)
                    fr = g / (r * r * r)
                elif same:
                    off = ~(r2 > 0.01)
                    r = torch.where(off, 1.0, r2).sqrt()
                    v = 1.0 / r
                    fr = v / (r * r)
                else:
                    off = r2 == 0.0
                    r = torch.where(off, 1.0, r2).sqrt()
                    e = torch.exp(-r / cfg.rs)
                    v = (1.0 - e) / r
                    fr = (1.0 / r - e * (1.0 / r + 1.0 / cfg.rs)) / (r * r)
                v = torch.where(off, 0.0, v)
                fr = torch.where(off, 0.0, fr)
                pot[part, sp] += 0.5 * sign * v.sum(1)
                for j in range(3):
                    force[part, j] += sign * (fr * d[j]).sum(1)
    return force.cpu().numpy(), pot.cpu().numpy()


def _exact_energies(pot, ne):
    # electrons' energy: every electron pair sum and the ions' share of e-i
    return pot[:ne].sum() + pot[ne:, 0].sum(), pot[ne:, 1].sum()


def _kinetic(x, v, m):
    r2 = (x * x).sum(1)
    xv = (x * v).sum(1)
    return m * (v * v).sum(), m * (xv * xv / r2).sum()


def _exact_loop(case, te, state, steps):
    x_el, v_el, f_el, x_ion, v_ion, f_ion = (a.copy() for a in state)
    me, mi = units.M_ELECTRON_AMU, units.M_ION_AMU
    for _ in range(steps):
        for x, v, f, m in ((x_el, v_el, f_el, me), (x_ion, v_ion, f_ion, mi)):
            v += 0.5 * DT * f / m
            x += DT * v
        f, pot = _exact_forces(case, te, x_el, x_ion)
        f_el, f_ion = f[:len(x_el)], f[len(x_el):]
        for v, f, m in ((v_el, f_el, me), (v_ion, f_ion, mi)):
            v += 0.5 * DT * f / m
    ee, ei = _exact_energies(pot, len(x_el))
    (ke, re), (ki, ri) = _kinetic(x_el, v_el, me), _kinetic(x_ion, v_ion, mi)
    return x_el, v_el, f_el, x_ion, v_ion, f_ion, (ee, ei, ke, ki, re, ri)


def exact(case, seed):
    n = case["n_el"] + case["n_ion"]
    seed = int(seed) * SEED_STRIDE % (1 << 31)
    if case["call"] == "ensemble":
        cl = _clouds(case, seed)
        if sum(float(len(c[0]) + len(c[3])) ** 2 for _, c in cl) > 7.5e10:
            return None
        got = [_exact_loop(case, te, c, case["steps"]) for te, c in cl]
        x, v, f = (np.vstack([np.vstack([g[k], g[k + 3]]) for g in got]) for k in range(3))
        return {"x": x, "v": v, "f": f, "sums": np.array([g[6] for g in got])}
    state = _plasma(case["n_el"], case["n_ion"], case["te"], seed)
    if case["call"] == "direct":
        rng = np.random.default_rng(seed)
        at = np.sort(rng.choice(n, min(case["targets"], n), replace=False))
        f, pot = _exact_forces(case, case["te"], state[0], state[3], at)
        return {"f": f, "epot": pot.sum(1)}
    if float(n) ** 2 * case["steps"] > 7.5e10:
        return None
    if case["call"] == "force":
        f, pot = _exact_forces(case, case["te"], state[0], state[3])
        ne = case["n_el"]
        out = {"f_el": f[:ne], "f_ion": f[ne:], "epot": np.array(_exact_energies(pot, ne))}
    else:
        got = _exact_loop(case, case["te"], state, case["steps"])
        out = dict(zip(("x_el", "v_el", "f_el", "x_ion", "v_ion", "f_ion"), got[:6]))
        out["sums"] = np.array(got[6])
    if case["rdf"]:
        # which pairs the walk sums directly is the tree's affair
        out["rdf_ei"], out["rdf_ii"] = None, None
    return out
