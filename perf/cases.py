"""The framework's own workloads as cases that can be timed and compared.

Every case goes through the public Python view of the C ABI (redgb.lib.System,
redgb.ensemble.Ensemble, redgb.proposer.Proposer).  Single-disk passes hand a state in
(rg_set_state, from pinned host records, as a code that couples to the integrator does), take
one or more steps through the main loop (rg_advance) and read the state back; a force pass is
one rg_calc_accel.  An ensemble pass advances every disk by a fixed number of attempts and
reads every disk's state.  The disks are the benchmark's: a star, giants, a swarm of
planetesimals or self-gravitating protoplanets, drawn here with numpy.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "red.cuda.closeencounter_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from redgb import bodies, lib, types as T  # noqa: E402
from redgb.ensemble import Ensemble  # noqa: E402
from redgb.proposer import Proposer  # noqa: E402

K = T.GAUSS
GIANTS = ((9.55e-4, 5.2, 0.05), (2.86e-4, 9.54, 0.05))
ROCKY = ((1.66e-7, 0.387, 0.2), (2.45e-6, 0.723, 0.007), (3.0e-6, 1.0, 0.017), (3.2e-7, 1.524, 0.093))
OUTER = ((4.37e-5, 19.2, 0.046), (5.15e-5, 30.07, 0.009))


# ------------------------------------------------------------------------------ cases

def listed():
    return [
        # A planetary system alone, the reference's smallest everyday run: star, four giants,
        # four rocky planets.  Latency and launches are all there is.
        dict(name="planets_rkf78_fp64", kind="step", integrator="rkf78", mode="fp64", n_gp=4, n_rp=4, n_pp=0, n_pl=0,
             n_tp=0, ring=False, hill=3.0, dt=2.5, tol=1e-10, steps=8),
        # The planetesimal-disk workload (1027 bodies, RKF7(8), encounters, collisions,
        # ejections on) in the bit-exact form: a user's long single-disk run, four steps of it.
        dict(name="planetesimal_disk_fp64", kind="step", integrator="rkf78", mode="fp64", n_gp=2, n_rp=0, n_pp=0,
             n_pl=1024, n_tp=0, ring=False, hill=3.0, dt=6.0, tol=1e-10, steps=4),
        # The same disk in mixed precision, one step.
        dict(name="planetesimal_disk_mixed", kind="step", integrator="rkf78", mode="mixed", n_gp=2, n_rp=0, n_pp=0,
             n_pl=1024, n_tp=0, ring=False, hill=3.0, dt=6.0, tol=1e-10, steps=1),
        # A few thousand self-gravitating protoplanets with giants, adaptive, an odd size:
        # the ordinary planet-formation run.
        dict(name="protoplanets_rkf78_fp64", kind="step", integrator="rkf78", mode="fp64", n_gp=2, n_rp=0, n_pp=2998,
             n_pl=0, n_tp=0, ring=False, hill=0.0, dt=4.0, tol=1e-10, steps=1),
        # The benchmark's headline: 16384 self-gravitating bodies, RK4 with a fixed step, in the
        # bit-exact form and in mixed precision.
        dict(name="self_gravitating_rk4_fp64", kind="step", integrator="rk4", mode="fp64", n_gp=0, n_rp=0, n_pp=16384,
             n_pl=0, n_tp=0, ring=False, hill=0.0, dt=0.1, tol=0.0, steps=1),
        dict(name="self_gravitating_rk4_mixed", kind="step", integrator="rk4", mode="mixed", n_gp=0, n_rp=0,
             n_pp=16384, n_pl=0, n_tp=0, ring=False, hill=0.0, dt=0.1, tol=0.0, steps=1),
        # One force evaluation with all three interaction blocks (self-interacting bodies,
        # planetesimals, test particles), the call of a user with an integrator of their own.
        dict(name="three_blocks_force_mixed", kind="force", mode="mixed", n_gp=2, n_rp=0, n_pp=1500, n_pl=1000,
             n_tp=777, ring=False),
        # The dense ring (131072 bodies and an embryo), RKF5 with encounters and collisions on:
        # the largest single disk, one step; and one bit-exact force evaluation of it.
        dict(name="dense_ring_rkf5_mixed", kind="step", integrator="rkf5", mode="mixed", n_gp=0, n_rp=0, n_pp=131072,
             n_pl=0, n_tp=0, ring=True, hill=3.0, dt=0.02, tol=1e-9, steps=1),
        dict(name="dense_ring_force_fp64", kind="force", mode="fp64", n_gp=0, n_rp=0, n_pp=131072, n_pl=0, n_tp=0,
             ring=True),
        # The batched ensemble: 256 disks of 512 to 8192 planetesimals in mixed precision, about
        # three years to the next output; and 64 such disks in the bit-exact form.
        dict(name="ensemble_mixed", kind="ensemble", mode="mixed", disks=256, n_lo=512, n_hi=8192, hill=3.0,
             attempts=128),
        dict(name="ensemble_fp64", kind="ensemble", mode="fp64", disks=64, n_lo=512, n_hi=8192, hill=3.0,
             attempts=40),
        # The step proposer on a training set: predictions, and the loss and its gradient.
        dict(name="proposer_gradient", kind="proposer", n=100000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("planets", "disk", "disk", "proto", "rk4", "rk4", "blocks", "ring", "ring_force", "ensemble",
                       "proposer"))
    mode = rng.choice(("fp64", "mixed"))
    base = dict(n_gp=2, n_rp=0, n_pp=0, n_pl=0, n_tp=0, ring=False)
    if kind == "planets":
        return dict(base, kind="step", integrator="rkf78", mode="fp64", n_gp=rng.randint(1, 4), n_rp=rng.randint(1, 4),
                    hill=3.0, dt=rng.uniform(2.0, 3.0), tol=1e-10, steps=rng.randint(2, 8))
    if kind == "disk":
        return dict(base, kind="step", integrator="rkf78", mode=mode, n_pl=_log(rng, 200, 20000), hill=3.0,
                    dt=rng.uniform(3.0, 6.0), tol=1e-10, steps=1)
    if kind == "proto":
        return dict(base, kind="step", integrator="rkf78", mode="fp64", n_pp=_log(rng, 100, 6000), hill=0.0,
                    dt=rng.uniform(2.0, 4.0), tol=1e-10, steps=1)
    if kind == "rk4":
        return dict(base, kind="step", integrator="rk4", mode=mode, n_gp=rng.randint(0, 2),
                    n_pp=_log(rng, 500, 30000), hill=0.0, dt=rng.uniform(0.05, 0.2), tol=0.0, steps=1)
    if kind == "blocks":
        return dict(base, kind="force", mode=mode, n_pp=_log(rng, 50, 5000), n_pl=_log(rng, 50, 5000),
                    n_tp=_log(rng, 20, 3000))
    if kind == "ring":
        return dict(base, kind="step", integrator="rkf5", mode="mixed", n_gp=0, n_pp=_log(rng, 8000, 120000),
                    ring=True, hill=3.0, dt=rng.uniform(0.01, 0.03), tol=1e-9, steps=1)
    if kind == "ring_force":
        return dict(base, kind="force", mode=mode, n_gp=0, n_pp=_log(rng, 4000, 100000), ring=True)
    if kind == "ensemble":
        return dict(kind="ensemble", mode=mode, disks=_log(rng, 8, 200 if mode == "mixed" else 60), n_lo=512,
                    n_hi=_log(rng, 1000, 8192), hill=3.0, attempts=rng.randint(20, 60))
    return dict(kind="proposer", n=_log(rng, 2000, 100000))


# ------------------------------------------------------------------------------ inputs

def _orbits(mu, a, e, inc, peri, node, mean):
    """Positions [AU] and velocities [AU/day] of orbital elements (vectorised)."""
    E = mean + e * np.sin(mean)
    for _ in range(12):
        E = E - (E - e * np.sin(E) - mean) / (1.0 - e * np.cos(E))
    ce, se, q = np.cos(E), np.sin(E), np.sqrt(1.0 - e * e)
    n = np.sqrt(mu / a) / (1.0 - e * ce)
    x, y, vx, vy = a * (ce - e), a * q * se, -n * se, n * q * ce
    cw, sw, cO, sO, ci, si = np.cos(peri), np.sin(peri), np.cos(node), np.sin(node), np.cos(inc), np.sin(inc)
    P = np.stack([cw * cO - sw * sO * ci, cw * sO + sw * cO * ci, sw * si], 1)
    Q = np.stack([-sw * cO - cw * sO * ci, -sw * sO + cw * cO * ci, cw * si], 1)
    return x[:, None] * P + y[:, None] * Q, vx[:, None] * P + vy[:, None] * Q


def _swarm(rng, n, ring, masses):
    """a, e, i, angles and masses of n small bodies: a surface density r^-1.5 on [1, 4] AU, or
    the ring's uniform [0.9, 1.1] AU."""
    u = rng.uniform(size=n)
    a = 0.9 + 0.2 * u if ring else (1.0 + u) ** 2
    s_e, s_i = (0.002, 0.002) if ring else (0.01, 0.005)
    e = np.minimum(rng.rayleigh(s_e, n), 0.9)
    inc = rng.rayleigh(s_i, n)
    ang = rng.uniform(0.0, 2.0 * math.pi, (3, n))
    m = np.exp(rng.uniform(math.log(masses[0]), math.log(masses[1]), n)) if masses else np.zeros(n)
    return a, e, inc, ang, m


def _disk(c, rng, scale=(1.0, 1.0)):
    """Arrays of one disk: counts, r, v, mass, radius, body type (the star at rest at 0)."""
    giants = [(m * s, a, e) for (m, a, e), s in zip(GIANTS, scale)] + list(OUTER)
    planets = giants[:c["n_gp"]] + list(ROCKY[:c["n_rp"]]) + ([(3e-6, 1.0, 0.0)] if c["ring"] else [])
    types = [T.BODY_GIANTPLANET] * c["n_gp"] + [T.BODY_ROCKYPLANET] * c["n_rp"] + [T.BODY_PROTOPLANET] * c["ring"]
    cols = [np.array(x, np.float64) for x in zip(*planets)] if planets else [np.zeros(0)] * 3
    n0 = len(planets)
    flat = 0.0 if not c["n_rp"] else 0.02  # the benchmark's giants are coplanar; a planetary system is not
    parts = [(cols[1], cols[2], rng.rayleigh(flat, n0), rng.uniform(0, 2 * math.pi, (3, n0)), cols[0])]
    parts.append(_swarm(rng, c["n_pp"], c["ring"], (1e-11, 1e-9) if c["ring"] else (1e-9, 1e-7)))
    parts.append(_swarm(rng, c["n_pl"], c["ring"], (1e-10, 1e-8)))
    parts.append(_swarm(rng, c["n_tp"], c["ring"], None))
    a, e, inc, m = (np.concatenate([p[k] for p in parts]) for k in (0, 1, 2, 4))
    peri, node, mean = np.concatenate([p[3] for p in parts], 1)
    r, v = _orbits(T.GAUSS2 * (1.0 + m), a, e, inc, peri, node, mean)
    typ = np.array([T.BODY_STAR] + types + [T.BODY_PROTOPLANET] * c["n_pp"] + [T.BODY_PLANETESIMAL] * c["n_pl"] +
                   [T.BODY_TESTPARTICLE] * c["n_tp"], np.int32)
    mass = np.concatenate([[1.0], m])
    rho = np.where(typ == T.BODY_PLANETESIMAL, 2.0, 1.33) * bodies.GRAM_PER_CM3_TO_SOLAR_PER_AU3
    radius = np.cbrt(mass / (bodies.FOUR_PI_OVER_THREE * rho))
    radius[0] = bodies.STAR_RADIUS_AU
    counts = (1, c["n_gp"], c["n_rp"], c["n_pp"] + int(c["ring"]), 0, c["n_pl"], c["n_tp"])
    z = np.zeros((1, 3))
    return counts, np.concatenate([z, r]), np.concatenate([z, v]), mass, radius, typ


def _records(r):
    out = np.zeros((len(r), 4))
    out[:, :3] = r
    return out


def _body_list(d):
    counts, r, v, mass, radius, typ = d
    n = len(mass)
    p, md = np.zeros(n, T.PARAM), np.zeros(n, T.BODY_MD)
    p["mass"], p["radius"] = mass, radius
    md["id"], md["body_type"] = np.arange(1, n + 1), typ
    return bodies.Disk(counts, _records(r).view(T.VEC).reshape(n), _records(v).view(T.VEC).reshape(n), p, md,
                       np.zeros(n), [])


def _ensemble_disks(c, seed):
    sizes = np.random.default_rng(1000 + c["disks"]).integers(c["n_lo"], c["n_hi"] + 1, c["disks"])
    rng = np.random.default_rng(seed)
    one = dict(n_gp=2, n_rp=0, n_pp=0, n_tp=0, ring=False)
    return [_disk(dict(one, n_pl=int(n)), rng, rng.uniform(0.5, 2.0, 2)) for n in sizes]


def _proposer_inputs(c, seed):
    rng = np.random.default_rng(seed)
    n = c["n"]
    x = np.stack([rng.normal(0.8, 0.4, n), rng.normal(0.0, 0.02, n), rng.normal(1.0, 0.03, n),
                  rng.normal(-0.37, 0.1, n), (rng.uniform(size=n) > 0.02).astype(np.float64),
                  rng.normal(0.0, 0.02, n), rng.normal(0.0, 0.02, n), rng.normal(0.0, 0.02, n)], 1).astype(np.float32)
    y = rng.normal(0.0, 0.02, n).astype(np.float32)
    w = np.concatenate([rng.normal(0, 0.35, 512), np.zeros(64), rng.normal(0, 0.15, 4096), np.zeros(64),
                        rng.normal(0, 0.1, 64), np.zeros(1)]).astype(np.float32)
    mean, std = x.mean(0), np.maximum(x.std(0), 1e-6).astype(np.float32)
    return x, y, w, mean, std


INTEGRATORS = {"rk4": T.INT_RK4, "rkf5": T.INT_RK5, "rkf78": T.INT_RKF78}


def prepare(case, seed):
    c = case
    if c["kind"] == "proposer":
        x, y, w, mean, std = _proposer_inputs(c, seed)
        net = Proposer(0)
        net.set_normalisation(mean, std)
        net.set_params(w)
        return dict(kind="proposer", net=net, x=x, y=y)
    mode = T.GRAVITY_FP64 if c["mode"] == "fp64" else T.GRAVITY_MIXED
    if c["kind"] == "ensemble":
        disks = [_body_list(d) for d in _ensemble_disks(c, seed)]
        ens = Ensemble(disks, bodies.thresholds())
        ens.set_integrator(dt_day=5.0, tolerance=1e-10)
        ens.set_options(gravity_mode=mode, hill_factor=c["hill"])
        n = sum(d.n_total for d in disks)
        return dict(kind="ensemble", ens=ens, attempts=c["attempts"], r=np.empty((n, 4)), v=np.empty((n, 4)),
                    t=np.empty(len(disks)))
    d = _disk(c, np.random.default_rng(seed))
    s = lib.System(_body_list(d), bodies.thresholds())
    s.set_gravity_mode(mode)
    if c["kind"] == "force":
        return dict(kind="force", sys=s)
    s.set_event_options(hill_factor=c["hill"])
    n = len(d[3])
    bufs = [torch.empty(n, 4, dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
    bufs[0][:], bufs[1][:] = _records(d[1]), _records(d[2])
    return dict(kind="step", sys=s, bufs=bufs, recs=[b.view(T.VEC).reshape(n) for b in bufs],
                integrator=INTEGRATORS[c["integrator"]], adaptive=c["integrator"] != "rk4", dt=c["dt"], tol=c["tol"],
                steps=c["steps"])


# ------------------------------------------------------------------------------ one pass

def run(state):
    s = state
    if s["kind"] == "force":
        a = s["sys"].calc_accel()
        return a.view(np.float64).reshape(len(a), 4)
    if s["kind"] == "proposer":
        pred = s["net"].forward(s["x"])
        grad, loss = s["net"].gradient(s["x"], s["y"])
        return dict(pred=pred, grad=grad, loss=np.float32(loss))
    if s["kind"] == "ensemble":
        ens, b = s["ens"], 0
        ens.advance(1e9, max_attempts=s["attempts"])
        for k in range(ens.n_sys):
            r, v, _, _, t = ens.state(k)
            n = len(r)
            s["r"][b:b + n] = r.view(np.float64).reshape(n, 4)
            s["v"][b:b + n] = v.view(np.float64).reshape(n, 4)
            s["t"][k] = t
            b += n
        ev, of = ens.events()
        return dict(r=s["r"], v=s["v"], t=s["t"], events=len(ev))
    g = s["sys"]
    g.set_state(*s["recs"][:2])
    g.set_integrator(s["integrator"], dt_day=s["dt"], adaptive=s["adaptive"], tolerance=s["tol"])
    steps = g.advance(1e12, max_steps=s["steps"])
    g.state(out=s["recs"][2:], params=False)
    ev = g.events()
    return dict(r=s["bufs"][2], v=s["bufs"][3], steps=steps, events=len(ev))


# ------------------------------------------------------------------------------ work

def _pairs(c, n_pl=None):
    si = 1 + c["n_gp"] + c["n_rp"] + c["n_pp"] + int(c["ring"])
    nsi, ni = c["n_pl"] if n_pl is None else n_pl, c["n_tp"]
    return si * (si + nsi - 1) + nsi * si + ni * (si + nsi), si + nsi + ni


def work(case):
    """36 flops per interacting pair (the reference's count) and evaluation; the state in and
    out (64 bytes a body each way), masses and radii, and for the ensemble, whose stage vectors
    do not fit the caches, the stage traffic of an attempt (93 vectors of 48 bytes a body)."""
    c = case
    if c["kind"] == "proposer":
        return {"bytes": c["n"] * 44.0 + 4801 * 8.0, "flops": c["n"] * 4 * 2.0 * 4672}
    if c["kind"] == "ensemble":
        mean_n = (c["n_lo"] + c["n_hi"]) / 2.0
        one = dict(n_gp=2, n_rp=0, n_pp=0, n_pl=0, n_tp=0, ring=False)
        pairs, n = _pairs(one, n_pl=mean_n)
        return {"bytes": c["disks"] * n * (c["attempts"] * 93 * 48.0 + 64.0),
                "flops": c["disks"] * c["attempts"] * (13 * 36.0 * pairs + 93 * 6 * 2.0 * n)}
    pairs, n = _pairs(c)
    if c["kind"] == "force":
        return {"bytes": 64.0 * n, "flops": 36.0 * pairs}
    evals = {"rk4": 4, "rkf5": 6, "rkf78": 13}[c["integrator"]] * c["steps"]
    vectors = {"rk4": 15, "rkf5": 27, "rkf78": 93}[c["integrator"]] * c["steps"]
    return {"bytes": 144.0 * n, "flops": 36.0 * pairs * evals + vectors * 12.0 * n}


# ------------------------------------------------------------------------------ 64 bits

def _accel(r, m, si, nm):
    """G = 1 accelerations of the three blocks: SI x massive, NSI x SI, NI x massive."""
    out = torch.zeros_like(r)
    n = r.shape[0]
    for lo, hi, src in ((0, si, nm), (si, nm, si), (nm, n, nm)):
        step = max(1, int(2.5e8) // max(src, 1))
        for a in range(lo, hi, step):
            b = min(hi, a + step)
            d = [r[None, :src, k] - r[a:b, k, None] for k in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            w = m[None, :src] / (r2 * r2.sqrt())
            w = torch.where(r2 == 0, torch.zeros_like(w), w)
            for k in range(3):
                out[a:b, k] = (w * d[k]).sum(1)
            del d, r2, w
    return out


_RK8_A = {
    1: {0: 2 / 27}, 2: {0: 1 / 36, 1: 1 / 12}, 3: {0: 1 / 24, 2: 1 / 8}, 4: {0: 5 / 12, 2: -25 / 16, 3: 25 / 16},
    5: {0: 1 / 20, 3: 1 / 4, 4: 1 / 5}, 6: {0: -25 / 108, 3: 125 / 108, 4: -65 / 27, 5: 125 / 54},
    7: {0: 31 / 300, 4: 61 / 225, 5: -2 / 9, 6: 13 / 900},
    8: {0: 2, 3: -53 / 6, 4: 704 / 45, 5: -107 / 9, 6: 67 / 90, 7: 3},
    9: {0: -91 / 108, 3: 23 / 108, 4: -976 / 135, 5: 311 / 54, 6: -19 / 60, 7: 17 / 6, 8: -1 / 12},
    10: {0: 2383 / 4100, 3: -341 / 164, 4: 4496 / 1025, 5: -301 / 82, 6: 2133 / 4100, 7: 45 / 82, 8: 45 / 164,
         9: 18 / 41},
    11: {0: 3 / 205, 5: -6 / 41, 6: -3 / 205, 7: -3 / 41, 8: 3 / 41, 9: 6 / 41},
    12: {0: -1777 / 4100, 3: -341 / 164, 4: 4496 / 1025, 5: -289 / 82, 6: 2193 / 4100, 7: 51 / 82, 8: 33 / 164,
         9: 12 / 41, 11: 1}}
_RK8_B = {0: 41 / 840, 5: 34 / 105, 6: 9 / 35, 7: 9 / 35, 8: 9 / 280, 9: 9 / 280, 10: 41 / 840}
_RK5_A = {1: {0: 1 / 5}, 2: {0: 3 / 40, 1: 9 / 40}, 3: {0: 3 / 10, 1: -9 / 10, 2: 6 / 5},
          4: {0: -11 / 54, 1: 5 / 2, 2: -70 / 27, 3: 35 / 27},
          5: {0: 1631 / 55296, 1: 175 / 512, 2: 575 / 13824, 3: 44275 / 110592, 4: 253 / 4096}}
_RK5_B = {0: 2825 / 27648, 2: 18575 / 48384, 3: 13525 / 55296, 4: 277 / 14336, 5: 1 / 4}
_RK4_A = {1: {0: 1 / 2}, 2: {1: 1 / 2}, 3: {2: 1.0}}
_RK4_B = {0: 1 / 6, 1: 1 / 3, 2: 1 / 3, 3: 1 / 6}


def exact(case, seed):
    c = case
    if c["kind"] == "ensemble":
        return None  # dozens of steps whose sizes follow each run's own rounding: no value to hold them to
    if c["kind"] == "proposer":
        return _exact_proposer(c, seed)
    counts, r, v, mass, _, _ = _disk(c, np.random.default_rng(seed))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = torch.tensor(mass, device=dev)
    si, nm = sum(counts[:4]), sum(counts[:6])
    f = lambda y: torch.cat([y[:, 3:], _accel(y[:, :3], m, si, nm)], 1)  # noqa: E731
    if c["kind"] == "force":
        # rg_create moves a disk whose star is at rest in the origin to its barycentre
        r = r - (mass[:, None] * r).sum(0) / mass.sum()
        return _records(_accel(torch.tensor(r, device=dev), m, si, nm).cpu().numpy())
    y = torch.tensor(np.concatenate([r, v / K], 1), device=dev)
    A, B = {"rk4": (_RK4_A, _RK4_B), "rkf5": (_RK5_A, _RK5_B), "rkf78": (_RK8_A, _RK8_B)}[c["integrator"]]
    dt = c["dt"] * K
    for _ in range(c["steps"]):
        k0 = f(y)
        while True:
            k = {0: k0}
            did = dt
            for s in sorted(A):
                k[s] = f(y + did * sum(q * k[p] for p, q in A[s].items()))
            new = y + did * sum(q * k[p] for p, q in B.items())
            if c["integrator"] != "rkf78":
                break  # a fixed step; the ring's trial step is far below what its tolerance takes
            e = (k[0] + k[10] - k[11] - k[12])[:nm].max().item()
            err = abs(did * 41 / 840 * max(e, 0.0))
            dt = did * 0.9 * (c["tol"] / err) ** (1 / 8)
            if err <= c["tol"]:
                break
        y = new
    y = y.cpu().numpy()
    return dict(r=_records(y[:, :3]), v=_records(y[:, 3:] * K), steps=None, events=None)


def _exact_proposer(c, seed):
    x, y, w, mean, std = _proposer_inputs(c, seed)
    z = torch.tensor((x - mean) / std, dtype=torch.float64)
    wb = torch.tensor(w).to(torch.bfloat16).double().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = wb.split([512, 64, 4096, 64, 64, 1])
    act = torch.nn.functional.silu
    h = act(act(z @ w1.view(64, 8).T + b1) @ w2.view(64, 64).T + b2)
    pred = h @ w3 + b3
    loss = (pred - torch.tensor(y, dtype=torch.float64)).square().mean()
    loss.backward()
    return dict(pred=pred.detach().numpy(), grad=wb.grad.numpy(), loss=float(loss))
