"""The certified FP64 form with a few bodies far outside the disk: an evaluation costs what it costs
without them, with the event screens on too, and the events are the oracle's."""
import numpy as np
import pytest

import pyoracle
from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu


def _disk(n, far, at):
    d = bodies.make_disk(n_pl=n, pl_type=T.BODY_PROTOPLANET, giants=(), seed=5, m_range=(1e-9, 1e-7))
    for k in range(far):  # pairs of neighbours far out
        i = 400 + 7 * k
        d.r["x"][i], d.r["y"][i], d.r["z"][i] = at + 5e-4 * (k % 2), 0.1 * (k // 2), 0.0
        d.v["x"][i], d.v["y"][i], d.v["z"][i] = 0.0, 0.5 * T.GAUSS / np.sqrt(at), 0.0
    return d


def _hill_ms(d, factor):
    """Time of the evaluations of a few RK4 steps, Hill log and (factor > 0) collisions on."""
    s = lib.System(d, bodies.thresholds(collision_factor=factor))
    s.set_event_options(hill_factor=3.0)
    s.set_integrator(T.INT_RK4, 0.01, False)
    best = np.inf
    for _ in range(4):
        s.step()
        s.set_profiling(True)
        a = s.profile()["gravity_ms"]
        for _ in range(2):
            s.step()
        best = min(best, s.profile()["gravity_ms"] - a)
        s.set_profiling(False)
    return best


def test_distant_bodies_leave_the_hill_screen_narrow(gpulib):
    """1000 AU out: the screen of every other body stays as wide as without them (with the
    largest star distance in it, the step took twice as long)."""
    whole, far = _hill_ms(_disk(4000, 0, 0.0), 0.0), _hill_ms(_disk(4000, 1, 1000.0), 0.0)
    assert far < 1.35 * whole, (whole, far)


@pytest.mark.parametrize("where", ["far", "high"])
def test_bodies_outside_the_grid_do_not_last_longest(gpulib, where):
    """A body 100 AU out, or 1 AU above the disk, has every pair taken exactly: by the row kernel, not by
    the one warp that has the sink (then the evaluations took more than twice as long)."""
    d = _disk(4000, 1 if where == "far" else 0, 100.0)
    if where == "high":
        d.r["z"][400] = 1.0
    whole, one = _hill_ms(_disk(4000, 0, 0.0), 1.0), _hill_ms(d, 1.0)
    assert one < 1.35 * whole, (whole, one)


@pytest.mark.parametrize("at", [30.0, 1000.0])
def test_events_with_distant_bodies(gpulib, at):
    d = _disk(2000, 6, at)
    thr = bodies.thresholds(ejection=0.0, collision_factor=60.0)
    got = []
    for s in (lib.System(d, thr), pyoracle.OracleSystem(d, thr)):
        s.set_integrator(T.INT_RK4, 0.01, False)
        s.set_event_options(hill_factor=3.0, close_encounter=True)
        s.advance(1e9, max_steps=2)
        got.append(s.events())
    assert len(got[0]) == len(got[1]) > 20
    ids = {tuple(sorted((int(e["id1"]), int(e["id2"])))) for e in got[1]}
    assert (401, 408) in ids and (429, 436) in ids  # far out
    for a, b in zip(*got):
        for f in T.EVENT.names:
            assert a[f] == b[f], (f, a, b)
