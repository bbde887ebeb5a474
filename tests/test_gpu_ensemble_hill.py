"""The ensemble's Hill-sphere log (ens_hill_kernel) against single disks: no pairs, some and more than
a warp's, over two steps so that the second finds its pairs among the first's; and a disk with more
pairs than its set holds is refused."""
import numpy as np
import pytest

from redgb import bodies, lib, types as T
from redgb.api import RedError
from redgb.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def test_hill_records_of_every_count(gpulib):
    sizes = (3, 40, 64, 65, 150)  # a disk of n planetesimals has up to 2 n pairs with its giants
    disks = [bodies.make_disk(n_pl=n, seed=n) for n in sizes]
    most = 0
    for hill in (3.0, 12.0, 20.0, 30.0):
        ens = Ensemble(disks, bodies.thresholds(collision_factor=0.0))
        ens.set_integrator(dt_day=1.0, tolerance=1e-10)
        ens.set_options(gravity_mode=T.GRAVITY_FP64, hill_factor=hill)
        ens.advance(1e9, max_attempts=2)
        ev, sys_of = ens.events()
        for k, d in enumerate(disks):
            s = lib.System(d, bodies.thresholds(collision_factor=0.0))
            s.set_integrator(T.INT_RKF78, 1.0, True, 1e-10)
            s.set_event_options(hill_factor=hill)
            while s.counters()["n_tried_step"] < 2:
                s.advance(1e9, max_steps=1)
            one = s.events()
            mine = ev[np.asarray(sys_of) == k]
            assert len(mine) == len(one), (hill, k)
            for f in ("event_name", "id1", "id2", "idx1", "idx2"):
                assert np.array_equal(mine[f], one[f]), (hill, k, f)
            most = max(most, len(one))
    assert most > 32


def test_more_pairs_than_a_set_holds(gpulib):
    disks = [bodies.make_disk(n_pl=n, seed=n) for n in (10, 1500)]
    ens = Ensemble(disks, bodies.thresholds(collision_factor=0.0))
    ens.set_integrator(dt_day=1.0, tolerance=1e-10)
    ens.set_options(gravity_mode=T.GRAVITY_FP64, hill_factor=90.0)
    with pytest.raises(RedError):
        ens.advance(1e9, max_attempts=2)
