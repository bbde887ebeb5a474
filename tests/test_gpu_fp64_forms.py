"""The FP64 forms of wide, shallow blocks (many sinks, a hundred sources or so) against the oracle, bit
for bit: single disks on both sides of the lines between rows, pair by pair and certified, with
planetesimals and test particles, and ensembles of small disks; with the event records."""
import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, lib, types as T
from redgb.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def _disk(si, pl, tp, seed=1):
    """A star, two giants, `si` protoplanets, `pl` planetesimals and `tp` test particles."""
    rng = np.random.RandomState(seed)
    emb = [(float(m), float(a), 0.01) for m, a in zip(np.exp(rng.uniform(np.log(1e-9), np.log(1e-7), si)),
                                                      1 + rng.uniform(size=si))]
    d = bodies.make_disk(n_pl=pl, seed=seed, embryos=emb, n_tp=tp, a_range=(1.0, 2.0))
    for f in "xyz":
        d.r[f][3:3 + si] += 0.003 * rng.normal(size=si)
    return d


def _sizes():
    # sinks on both sides of the line to rows, tiles of 4 to 32 sinks with one over, sources around the tiles' 32 to 256
    return [(62, 0, 511), (62, 0, 512), (62, 1501, 0), (62, 0, 4801), (70, 700, 701), (125, 0, 1537), (126, 2000, 33),
            (200, 0, 1073), (200, 1074, 1075), (200, 0, 8391), (200, 0, 8392), (253, 0, 1700), (254, 1333, 0), (400, 0, 2160)]


@pytest.mark.parametrize("si,pl,tp", _sizes())
def test_accelerations_bit_exact(gpulib, si, pl, tp):
    d = _disk(si, pl, tp)
    d.md["id"][20] *= -1
    d.md["id"][40] = 0
    d.p["mass"][30] = 0.0
    ag = lib.System(d, bodies.thresholds()).calc_accel()
    ao = pyoracle.OracleSystem(d, bodies.thresholds()).calc_accel()
    for f in "xyz":
        assert H.same(ag[f], ao[f]), (f, int((ag[f] != ao[f]).sum()))


@pytest.mark.parametrize("si,pl,tp", [(70, 900, 901), (100, 3000, 1500)])
def test_events_match_oracle(gpulib, si, pl, tp):
    d = _disk(si, pl, tp)
    for q in range(4):  # planetesimals and test particles beside protoplanets
        for j, i in ((3 + si + 7 * q, 10 + q), (3 + si + pl + 5 * q, 20 + q)):
            for f in "xyz":
                d.r[f][j], d.v[f][j] = d.r[f][i], d.v[f][i]
            d.r["x"][j] += 1e-6 * (1 + q)
    thr = bodies.thresholds(collision_factor=1.0)
    got = []
    for s in (lib.System(d, thr), pyoracle.OracleSystem(d, thr)):
        s.set_integrator(T.INT_RK4, 0.5, False)
        s.set_event_options(hill_factor=3.0)
        s.advance(1e9, max_steps=2)
        got.append((s.events(), s.state(internal=True)))
    (eg, sg), (eo, so) = got
    assert len(eg) == len(eo) > 5
    for a, b in zip(eg, eo):
        for f in T.EVENT.names:
            assert a[f] == b[f], (f, a, b)
    for a, b in zip(sg[:2], so[:2]):
        for f in "xyz":
            assert H.same(a[f], b[f]), f


def test_steps_with_all_forms(gpulib):
    """RKF7(8) attempts from a graph, with rows, a block pair by pair and a certified one on two streams."""
    d, thr = _disk(100, 2000, 1200), bodies.thresholds()
    got = []
    for s in (lib.System(d, thr), pyoracle.OracleSystem(d, thr)):
        s.set_integrator(T.INT_RKF78, 1.0, True, 1e-10)
        s.set_event_options(hill_factor=3.0)
        s.advance(1e9, max_steps=3)
        got.append(s.state(internal=True))
    for a, b in zip(got[0][:2], got[1][:2]):
        for f in "xyz":
            assert H.same(a[f], b[f]), f


# disks x (protoplanets, planetesimals, test particles): blocks of many sinks pair by pair; few heavy rows
# pair by pair; short rows with them; heavy rows of certified disks; mixed sizes
ENSEMBLES = {"protoplanets": [(100, 0, 0)] * 20, "few": [(0, 90, 0)] * 300, "short_rows": [(100, 0, 900)] * 3,
             "certified": [(240, 0, 0)] * 60, "sizes": [(62, 40, 70), (150, 0, 33), (0, 300, 5), (30, 100, 100)] * 8}


@pytest.mark.parametrize("name", list(ENSEMBLES))
def test_ensembles_bit_exact(gpulib, name):
    kinds = ENSEMBLES[name]
    one = {k: _disk(*k, seed=3) for k in set(kinds)}
    thr = bodies.thresholds()
    e = Ensemble([one[k] for k in kinds], thr)
    e.set_integrator(2.0, 1e-10)
    e.set_options(gravity_mode=T.GRAVITY_FP64, hill_factor=0.0)
    e.advance(1e9, max_attempts=1)  # (the next trial step is the device's pow, not the oracle's)
    for k in one:
        last = len(kinds) - 1 - kinds[::-1].index(k)
        passed = e.stats(last)["n_passed_step"]
        assert passed == 1
        o = pyoracle.OracleSystem(one[k], thr)
        o.set_integrator(T.INT_RKF78, 2.0, True, 1e-10)
        o.advance(1e9, max_steps=passed)
        ro, vo = o.state()[:2]
        for s in (kinds.index(k), last):
            rg, vg = e.state(s)[:2]
            for f in "xyz":
                assert H.same(rg[f], ro[f]) and H.same(vg[f], vo[f]), (k, s, f)
