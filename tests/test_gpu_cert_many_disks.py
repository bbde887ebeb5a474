"""The certified FP64 form over more disks than a grid has rows (65 535): the first, the 65 536th and
the last disk of such an ensemble against the oracle, bit for bit."""
import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, types as T
from redgb.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def test_more_disks_than_grid_rows(gpulib):
    d = bodies.make_disk(n_pl=64, pl_type=T.BODY_PROTOPLANET, giants=(), seed=4, m_range=(1e-9, 1e-7))
    thr = bodies.thresholds()
    n = 65537
    e = Ensemble([d] * n, thr)
    e.set_integrator(0.5, 1e-10)
    e.set_options(gravity_mode=T.GRAVITY_FP64, hill_factor=0.0)
    e.advance(1e9, max_attempts=1)
    o = pyoracle.OracleSystem(d, thr)
    o.set_integrator(T.INT_RKF78, 0.5, True, 1e-10)
    o.advance(1e9, max_steps=1)
    ro, vo = o.state()[:2]
    for k in (0, 65535, n - 1):
        rg, vg = e.state(k)[:2]
        for f in "xyz":
            assert H.same(rg[f], ro[f]) and H.same(vg[f], vo[f]), (k, f)
