"""Heavy rows whose sums go through zero at every other term (planetesimals in antipodal pairs, one after
the other): the oracle's bits in every kernel that adds such rows, and no more than a few times an
ordinary disk's time."""
import time

import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, lib, types as T
from redgb.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def _pairs(n, kind=T.BODY_PLANETESIMAL):
    d = bodies.make_disk(n_pl=n, pl_type=kind, seed=2, m_range=(1e-9, 1e-7))
    even, odd = slice(3, 3 + n // 2 * 2, 2), slice(4, 3 + n // 2 * 2, 2)
    for f in "xyz":
        d.r[f][odd], d.v[f][odd] = -d.r[f][even], -d.v[f][even]
    d.p["mass"][odd] = d.p["mass"][even]
    return d


def _same(a, b):
    for f in "xyz":
        assert H.same(a[f], b[f]), (f, int((a[f] != b[f]).sum()))


@pytest.mark.parametrize("n,kind", [(60, T.BODY_PLANETESIMAL), (301, T.BODY_PLANETESIMAL), (1153, T.BODY_PLANETESIMAL),
                                    (4000, T.BODY_PLANETESIMAL), (500, T.BODY_PROTOPLANET), (2000, T.BODY_PROTOPLANET)])
def test_bits(gpulib, n, kind):
    d = _pairs(n, kind)
    thr = bodies.thresholds()
    _same(lib.System(d, thr).calc_accel(), pyoracle.OracleSystem(d, thr).calc_accel())


@pytest.mark.parametrize("n", [301, 1000])
def test_step_bits(gpulib, n):
    d, thr = _pairs(n), bodies.thresholds()
    s, o, e = lib.System(d, thr), pyoracle.OracleSystem(d, thr), Ensemble([d, d], thr)
    for x in (s, o):
        x.set_integrator(T.INT_RKF78, 0.5, True, 1e-10)
        x.advance(1e9, max_steps=1)
    e.set_integrator(0.5, 1e-10)
    e.set_options(gravity_mode=T.GRAVITY_FP64, hill_factor=0.0)
    e.advance(1e9, max_attempts=1)
    for a in (s.state(), e.state(1)):
        for q in (0, 1):
            _same(a[q], o.state()[q])


def test_time(gpulib):
    """A chain a row: four times an ordinary disk's attempt; every lane's segment added again took ten."""
    def us(d):
        s = lib.System(d, bodies.thresholds())
        s.set_integrator(T.INT_RKF78, 0.01, False)
        s.advance(1e9, max_steps=2)
        best = np.inf
        for _ in range(5):
            t0 = time.perf_counter()
            s.advance(1e9, max_steps=4)
            best = min(best, time.perf_counter() - t0)
        return best / 4
    ordinary = us(bodies.make_disk(n_pl=1000, seed=2, m_range=(1e-9, 1e-7)))
    assert us(_pairs(1000)) < 6.5 * ordinary
