"""The FP64 gravity whose pair terms are certified integers (csrc/gravity_cert.cu) and the row
kernel beside it (csrc/gravity_fp64.cu) against the oracle, bit for bit: block sizes on both
sides of the line between the two, ragged epochs, and states that the approximation has to
hand over -- coplanar and tall disks, near pairs, sums that hover, masses and coordinates
outside the splits' range, inactive, massless and NaN bodies -- with the event records."""
import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu


def _disk(kind):
    d = bodies.make_disk(n_pl=1900, pl_type=T.BODY_PROTOPLANET, seed=5, m_range=(1e-9, 1e-7))
    rng = np.random.RandomState(3)
    if kind == "coplanar":
        d.r["z"] = 0.0
    elif kind == "tall":
        d.r["z"] *= 1e3
    elif kind == "heavy":
        d.p["mass"][3:] = np.exp(rng.uniform(np.log(1e-6), np.log(1e-3), 1900))
    elif kind == "light":
        d.p["mass"][3:] = np.exp(rng.uniform(np.log(1e-45), np.log(1e-18), 1900))
    elif kind == "cluster":
        for f in "xyz":
            d.r[f] = rng.normal(size=d.n_total)
        d.p["mass"] = 1e-3
    elif kind == "strange":
        d.r["x"][700], d.p["mass"][700] = 1e20, 0.0   # a parked merger
        d.r["x"][800], d.r["y"][900] = 1e17, 9e4      # far bodies with mass
        d.md["id"][30] *= -1
        d.md["id"][500] = 0
        d.p["mass"][1000] = 0.0
        for f in "xyz":
            d.r[f][100:120] = d.r[f][200] + 1e-7 * rng.normal(size=20)
    elif kind == "coincident":
        d.r[100] = d.r[101]
    elif kind == "nan":
        d.r["y"][1500] = np.nan
    elif kind == "blocks":
        d = bodies.make_disk(n_pl=900, seed=9, embryos=[(1e-7, 1.0 + 0.0015 * k, 0.01) for k in range(1900)], n_tp=1300)
        d.r["z"][3:1903] = 0.003 * rng.normal(size=1900)
    return d


KINDS = ["ordinary", "coplanar", "tall", "heavy", "light", "cluster", "strange", "coincident", "nan", "blocks"]


@pytest.mark.parametrize("kind", KINDS)
def test_accelerations_bit_exact(gpulib, kind):
    d = _disk(kind)
    ag = lib.System(d, bodies.thresholds()).calc_accel()
    ao = pyoracle.OracleSystem(d, bodies.thresholds()).calc_accel()
    for f in "xyz":
        assert H.same(ag[f], ao[f]), (kind, f, int((ag[f] != ao[f]).sum()))


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 255, 1151, 1153, 1785, 1790, 2049, 2305])
def test_block_sizes_bit_exact(gpulib, n):
    """Single rows, a head without an epoch, row chunks and epochs with one body over, and both
    sides of the line between the row kernel and the certified one."""
    d = bodies.make_disk(n_pl=n, pl_type=T.BODY_PROTOPLANET, giants=(), seed=n, m_range=(1e-9, 1e-7))
    ag = lib.System(d, bodies.thresholds()).calc_accel()
    ao = pyoracle.OracleSystem(d, bodies.thresholds()).calc_accel()
    for f in "xyz":
        assert H.same(ag[f], ao[f]), (n, f)


def test_events_of_a_step_match_oracle(gpulib):
    """Collisions and Hill encounters found beside the certified terms: the oracle's records."""
    d = bodies.make_disk(n_pl=2000, pl_type=T.BODY_PROTOPLANET, seed=11, m_range=(1e-9, 1e-7), a_range=(1.0, 1.6))
    thr = bodies.thresholds(collision_factor=40.0)
    got = []
    for s in (lib.System(d, thr), pyoracle.OracleSystem(d, thr)):
        s.set_integrator(T.INT_RK4, 0.5, False)
        s.set_event_options(hill_factor=3.0)
        s.advance(1e9, max_steps=2)
        got.append((s.events(), s.state(internal=True)))
    (eg, sg), (eo, so) = got
    assert len(eg) == len(eo) > 20
    for a, b in zip(eg, eo):
        for f in T.EVENT.names:
            assert a[f] == b[f], (f, a, b)
    for a, b in zip(sg[:2], so[:2]):
        for f in "xyz":
            assert H.same(a[f], b[f]), f
