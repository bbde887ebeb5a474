"""RKF7(8) steps of small systems, each attempt one kernel (csrc/small_step.cu), against the oracle
bit for bit: 1 to 32 bodies (and 33, the first size on the other path), every mix of
interaction blocks, with and without step-size control, rejected attempts, and the events --
collisions, Hill encounters, ejections, hit-star."""
import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu


def _pair(disk, thr, adaptive=True, tol=1e-10, dt=1.0, hill=3.0, ectp=False):
    out = []
    for s in (lib.System(disk, thr), pyoracle.OracleSystem(disk, thr)):
        s.set_integrator(T.INT_RKF78, dt, adaptive, tol, ectp)
        s.set_event_options(hill_factor=hill)
        out.append(s)
    return out


def _same(g, o):
    a, b = g.state(internal=True), o.state(internal=True)
    assert a[4] == b[4]
    for k in (0, 1):
        for f in "xyz":
            assert H.same(a[k][f], b[k][f]), f
    assert np.array_equal(a[3]["id"], b[3]["id"])
    assert H.same(a[2]["mass"], b[2]["mass"])
    ga, gb = g.counters(), o.counters()
    for f in ("n_failed_step", "n_passed_step", "n_tried_step"):
        assert ga[f] == gb[f]
    eg, eo = g.events(), o.events()
    assert len(eg) == len(eo)
    for x, y in zip(eg, eo):
        for f in T.EVENT.names:
            assert x[f] == y[f], f
    return len(eg)


def _disk(n_emb, n_pl, n_tp, seed, scale=1.0):
    return bodies.make_disk(n_pl=n_pl, n_tp=n_tp, seed=seed, m_range=(1e-7, 1e-5),
                            embryos=[(1e-6, (1.0 + 0.2 * k) * scale, 0.05) for k in range(n_emb)])


@pytest.mark.parametrize("shape", [(0, 0, 0), (1, 0, 0), (6, 0, 0), (29, 0, 0), (30, 0, 0), (0, 29, 0), (0, 0, 29),
                                   (5, 8, 3), (0, 1, 28), (20, 5, 4)])
@pytest.mark.parametrize("adaptive", [True, False])
def test_small_systems_bit_exact(gpulib, shape, adaptive):
    d = _disk(*shape, seed=sum(shape) + 1)
    g, o = _pair(d, bodies.thresholds(), adaptive, dt=2.0, ectp=shape[2] > 5)
    for _ in range(3):
        g.advance(1e9, max_steps=4)
        o.advance(1e9, max_steps=4)
        _same(g, o)


def test_single_star(gpulib):
    d = bodies.make_disk(n_pl=0, giants=(), seed=1)
    g, o = _pair(d, bodies.thresholds(), adaptive=False)
    g.advance(1e9, max_steps=2)
    o.advance(1e9, max_steps=2)
    _same(g, o)


def test_rejected_attempts(gpulib):
    d = _disk(3, 4, 0, seed=2)
    g, o = _pair(d, bodies.thresholds(), dt=60.0, tol=1e-12)  # far too long a first trial step
    for s in (g, o):
        s.advance(1e9, max_steps=5)
    assert o.counters()["n_failed_step"] > 0
    _same(g, o)


@pytest.mark.parametrize("factor,steps", [(200.0, 600), (30.0, 200)])
def test_events(gpulib, factor, steps):
    """Collisions with compaction and an ejection; ejections and a hit-star event."""
    d = _disk(10, 12, 4, seed=5, scale=0.3)
    d.v["x"][3:7] *= 4.0  # unbound
    g, o = _pair(d, bodies.thresholds(ejection=6.0, hit_centrum=0.25, collision_factor=factor), dt=1.0, tol=1e-9)
    seen = 0
    for _ in range(steps // 10):
        for s in (g, o):
            s.advance(1e9, max_steps=10)
        seen += _same(g, o)
    c = o.counters()
    assert seen > 3 and c["n_ejection"][0] > 0
    assert (c["n_collision"][0] > 3 and o.n_total()[1] < 29) if factor > 100 else c["n_hit_centrum"][0] > 0


def test_set_state_between_steps(gpulib):
    """A state handed in is screened for ejections although the step before found none."""
    d = _disk(4, 3, 0, seed=8)
    g, o = _pair(d, bodies.thresholds(ejection=100.0), dt=1.0)
    for s in (g, o):
        s.advance(1e9, max_steps=2)
        r, v = s.state()[:2]
        r["x"][4] = 150.0
        s.set_state(r, v)
        s.advance(1e9, max_steps=1)
    assert _same(g, o) >= 1
