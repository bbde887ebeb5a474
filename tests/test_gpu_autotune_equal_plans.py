"""Where the sinks per tile shape nothing of the FP64 plan, the tuners leave them as they were."""
import pytest

from redgb import bodies, lib, types as T
from redgb.ensemble import Ensemble

pytestmark = pytest.mark.gpu


def test_equal_plans_keep_the_default(gpulib):
    d = bodies.make_disk(n_pl=300, pl_type=T.BODY_PROTOPLANET, giants=(), seed=2, m_range=(1e-9, 1e-7))
    for _ in range(6):  # (a row each: no certified tiles)
        assert lib.System(d, bodies.thresholds()).autotune(reps=1)["pairpar_sinks"] == 16
        e = Ensemble([d, d], bodies.thresholds())
        e.set_integrator(1.0, 1e-10)
        assert e.autotune(reps=1)["pairpar_sinks"] == 16
