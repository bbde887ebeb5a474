"""RKF7(8) steps of planetesimal disks in mixed precision, each attempt one cluster kernel
(csrc/swarm_step.cu), against the same steps as separate kernels (taken while timing hooks are
on): slices that are full, partial and empty, one to four heavy bodies, rejected attempts,
collisions, Hill encounters, ejections, and the first size beyond the cluster.

The separate kernels' segments are the cluster's slices, so every bit agrees: state, step sizes,
events."""
import numpy as np
import pytest

import helpers as H
from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu

GIANTS = ((9.55e-4, 5.2, 0.05), (2.86e-4, 9.54, 0.05), (4.4e-5, 19.2, 0.05))


def _pair(disk, thr, adaptive, dt, tol=1e-10, hill=3.0, ectp=False):
    out = []
    for general in (False, True):
        s = lib.System(disk, thr)
        s.set_gravity_mode(T.GRAVITY_MIXED)
        s.set_integrator(T.INT_RKF78, dt, adaptive, tol, ectp)
        s.set_event_options(hill_factor=hill)
        if general:
            s.set_profiling(1)
        out.append(s)
    return out


def _same(g, o):
    a, b = g.state(internal=True), o.state(internal=True)
    assert a[4] == b[4]
    for k in (0, 1):
        for f in "xyz":
            assert H.same(a[k][f], b[k][f]), f
    assert np.array_equal(a[3]["id"], b[3]["id"])
    ca, cb = g.counters(), o.counters()
    for f in ("n_failed_step", "n_passed_step", "n_tried_step", "n_gravity_evals"):
        assert ca[f] == cb[f]
    ea, eb = g.events(), o.events()
    assert len(ea) == len(eb)
    for f in T.EVENT.names:
        assert np.array_equal(ea[f], eb[f]), f
    return len(ea)


@pytest.mark.parametrize("n_pl", [64, 65, 95, 256, 257, 511, 513, 1024, 3071, 3072, 3073])
@pytest.mark.parametrize("n_giants", [0, 2, 3])
def test_fixed_steps(gpulib, n_pl, n_giants):
    d = bodies.make_disk(n_pl=n_pl, giants=GIANTS[:n_giants], giant_scale=(1.0,) * 3, seed=n_pl + n_giants)
    g, o = _pair(d, bodies.thresholds(), False, 4.0)
    for s in (g, o):
        s.advance(1e9, max_steps=3)
    _same(g, o)


@pytest.mark.parametrize("n_pl,ectp", [(100, False), (400, True), (1500, False), (3000, True)])
def test_adaptive_steps_with_events(gpulib, n_pl, ectp):
    """A first step of 60 days is rejected; radii grown so that bodies collide and merge."""
    d = bodies.make_disk(n_pl=n_pl, giants=GIANTS[:2], seed=7, m_range=(1e-9, 1e-7))
    d.p["radius"][1:] *= 400.0
    for k in range(4):  # started next to a giant: a collision and a Hill encounter
        for f, off in zip("xyz", (0.02 + 0.03 * k, 0.01, 0.0)):
            d.r[f][10 + k] = d.r[f][1] + off
            d.v[f][10 + k] = d.v[f][1]
    g, o = _pair(d, bodies.thresholds(ejection=30.0), True, 60.0, ectp=ectp)
    n = 0
    for _ in range(3):
        for s in (g, o):
            s.advance(1e9, max_steps=3)
        n += _same(g, o)
    assert n > 0 and g.counters()["n_failed_step"] > 0
