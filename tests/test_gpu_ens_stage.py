"""A stage of the ensemble's mixed-precision attempt in one kernel (csrc/ens_stage.cu) against the
same stages as separate kernels (taken while timing hooks are on), bit for bit: one to three heavy
bodies, segments that start and end inside disks, merged bodies, rejected attempts and collisions;
and a batch with a disk that keeps the separate kernels."""
import numpy as np
import pytest

import helpers as H
from redgb import bodies, types as T
from redgb.ensemble import Ensemble

pytestmark = pytest.mark.gpu

GIANTS = ((9.55e-4, 5.2, 0.05), (2.86e-4, 9.54, 0.05), (4.4e-5, 19.2, 0.05))


def _run(disks, general, attempts, factor):
    ens = Ensemble(disks, bodies.thresholds(collision_factor=factor))
    ens.set_integrator(dt_day=40.0, tolerance=1e-10)
    ens.set_options(gravity_mode=T.GRAVITY_MIXED, hill_factor=3.0)
    if general:
        ens.set_profiling(True)
    ens.advance(1e9, max_attempts=attempts)
    return [ens.state(k) for k in range(len(disks))], ens.events(), [ens.stats(k) for k in range(len(disks))]


def _same(disks, attempts=12, factor=1.0):
    a, ea, sa = _run(disks, False, attempts, factor)
    b, eb, sb = _run(disks, True, attempts, factor)
    for x, y in zip(a, b):
        assert x[4] == y[4]
        for k in (0, 1):
            for f in "xyz":
                assert H.same(x[k][f], y[k][f]), f
    assert len(ea[0]) == len(eb[0])
    for f in T.EVENT.names:
        assert np.array_equal(ea[0][f], eb[0][f]), f
    assert sa == sb
    return len(ea[0]), sum(s["n_failed_step"] for s in sa)


def test_uneven_disks(gpulib):
    sizes = (70, 255, 256, 257, 1000, 3000, 512, 130, 2049)
    disks = [bodies.make_disk(n_pl=n, giants=GIANTS[:n % 3], giant_scale=(1.0,) * 3, seed=n) for n in sizes]
    _, failed = _same(disks)
    assert failed > 0


def test_collisions(gpulib):
    disks = []
    for n in (100, 700, 1500):
        d = bodies.make_disk(n_pl=n, giants=GIANTS[:2], seed=n)
        for k in range(4):  # next to a giant
            for f, off in zip("xyz", (0.004 + 0.01 * k, 0.003, 0.0)):
                d.r[f][10 + k] = d.r[f][1] + off
                d.v[f][10 + k] = d.v[f][1]
        disks.append(d)
    n, _ = _same(disks, factor=50.0)
    assert n > 0


def test_batch_with_another_kind(gpulib):
    disks = [bodies.make_disk(n_pl=300, seed=1), bodies.make_disk(n_pl=200, seed=2, n_tp=40)]
    _same(disks)
