"""The certified FP64 gravity's two warp shapes (two sinks a warp below ten warps an SM, four above),
the row kernel's two (around rows of 384 and 448 sources) and the line between the kernels, against
the oracle bit for bit."""
import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu


def _same(d):
    ag = lib.System(d, bodies.thresholds()).calc_accel()
    ao = pyoracle.OracleSystem(d, bodies.thresholds()).calc_accel()
    for f in "xyz":
        assert H.same(ag[f], ao[f]), (f, int((ag[f] != ao[f]).sum()))


@pytest.mark.parametrize("n", [383, 384, 447, 448, 1498, 1500, 6063, 6079, 6080, 6095, 7001])
def test_sizes(gpulib, n):
    _same(bodies.make_disk(n_pl=n, pl_type=T.BODY_PROTOPLANET, giants=(), seed=n, m_range=(1e-9, 1e-7)))


@pytest.mark.parametrize("kind", ["coplanar", "tall", "cluster", "strange"])
def test_four_sinks_a_warp(gpulib, kind):
    """States that the approximation has to hand over, at a size of the second shape."""
    d = bodies.make_disk(n_pl=6400, pl_type=T.BODY_PROTOPLANET, seed=5, m_range=(1e-9, 1e-7))
    rng = np.random.RandomState(3)
    if kind == "coplanar":
        d.r["z"] = 0.0
    elif kind == "tall":
        d.r["z"] *= 1e3
    elif kind == "cluster":
        for f in "xyz":
            d.r[f] = rng.normal(size=d.n_total)
        d.p["mass"] = 1e-3
    else:
        d.r["x"][700], d.p["mass"][700] = 1e20, 0.0   # a parked merger
        d.r["x"][800], d.r["y"][900] = 1e17, 9e4      # far bodies with mass
        d.md["id"][30] *= -1
        d.md["id"][500] = 0
        d.p["mass"][1000] = 0.0
        for f in "xyz":
            d.r[f][100:120] = d.r[f][200] + 1e-7 * rng.normal(size=20)
    _same(d)
