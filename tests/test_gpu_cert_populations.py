"""The certified FP64 form on disks of two populations (bodies far out among the disk's, a few high orbits
over a flat or a thin disk), where many pairs or sums are not for its integers: bits and events against
the oracle, and the time of an evaluation beside an ordinary disk's."""
import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu


def _disk(n, kind, share, seed=4):
    d = bodies.make_disk(n_pl=n, pl_type=T.BODY_PROTOPLANET, seed=seed, m_range=(1e-9, 1e-7))
    rng = np.random.RandomState(seed)
    at = 3 + rng.permutation(n)[:int(n * share)]
    if kind == "far":
        f = np.exp(rng.uniform(np.log(5), np.log(1500), len(at)))
        for q in "xyz":
            d.r[q][at] *= f
            d.v[q][at] /= np.sqrt(f)
    elif kind == "flat":  # all others exactly in the plane
        z = d.r["z"].copy()
        d.r["z"], d.v["z"] = 0.0, 0.0
        d.r["z"][at] = 3 * z[at]
    elif kind == "thin":
        d.r["z"] *= 1e-4
        d.v["z"] *= 1e-4
        d.r["z"][at] = 0.1 * rng.normal(size=len(at))
    return d


@pytest.mark.parametrize("share", [0.02, 0.1, 0.4])
@pytest.mark.parametrize("kind", ["far", "flat", "thin"])
def test_bits(gpulib, kind, share):
    d = _disk(2500, kind, share)
    ag = lib.System(d, bodies.thresholds()).calc_accel()
    ao = pyoracle.OracleSystem(d, bodies.thresholds()).calc_accel()
    for f in "xyz":
        assert H.same(ag[f], ao[f]), (f, int((ag[f] != ao[f]).sum()))


@pytest.mark.parametrize("kind", ["far", "flat", "thin"])
def test_events(gpulib, kind):
    d = _disk(1800, kind, 0.2)
    for k in range(12):  # neighbours, some of either population
        i, j = 100 + 90 * k, 1500 + 11 * k
        for f in "xyz":
            d.r[f][j], d.v[f][j] = d.r[f][i], d.v[f][i]
        d.r["x"][j] += 2e-6 * (1 + k)
    thr = bodies.thresholds(ejection=0.0, collision_factor=1.0)
    got = []
    for s in (lib.System(d, thr), pyoracle.OracleSystem(d, thr)):
        s.set_integrator(T.INT_RK4, 0.01, False)
        s.set_event_options(hill_factor=3.0)
        for _ in range(2):
            s.step()
            s.check_for_collision()
        got.append((s.events(), s.state(internal=True)))
    (eg, sg), (eo, so) = got
    assert len(eg) == len(eo) > 5
    for a, b in zip(eg, eo):
        for f in T.EVENT.names:
            assert a[f] == b[f], (f, a, b)
    for a, b in zip(sg[:2], so[:2]):
        for f in "xyz":
            assert H.same(a[f], b[f]), f


def _ms(d):
    """Time of a step's four evaluations, collisions on."""
    s = lib.System(d, bodies.thresholds(ejection=0.0, collision_factor=1.0))
    s.set_integrator(T.INT_RK4, 0.001, False)
    for _ in range(2):
        s.step()
    s.set_profiling(True)
    best = np.inf
    for _ in range(3):
        a = s.profile()["gravity_ms"]
        s.step()
        best = min(best, s.profile()["gravity_ms"] - a)
    return best


@pytest.mark.parametrize("kind,share", [("far", 0.3), ("flat", 0.1), ("thin", 0.1)])
def test_time(gpulib, kind, share):
    """Every pair by the row kernel costs three and a half times an ordinary disk's evaluation; taken in
    the certified kernel's single warps these states cost nine times as much."""
    whole, two = _ms(_disk(8000, kind, 0.0)), _ms(_disk(8000, kind, share))
    assert two < 5.0 * whole, (whole, two)
