"""RKF7(8) steps of planetesimal disks in FP64, each attempt one cluster kernel
(csrc/swarm_fp64.cu), bit for bit against the oracle and, over every kind of slice, against the
same steps as separate kernels (taken while timing hooks are on); and the CTA's row sum
(cta_row_sum, csrc/row_sum.h) against the serial sum."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

import helpers as H
import pyoracle
from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu

GIANTS = ((9.55e-4, 5.2, 0.05), (2.86e-4, 9.54, 0.05), (4.4e-5, 19.2, 0.05))


def _start(s, adaptive, dt, hill=3.0, ectp=False):
    s.set_integrator(T.INT_RKF78, dt, adaptive, 1e-10, ectp)
    s.set_event_options(hill_factor=hill)
    return s


def _same(g, o):
    a, b = g.state(internal=True), o.state(internal=True)
    assert a[4] == b[4]
    for k in (0, 1):
        for f in "xyz":
            assert H.same(a[k][f], b[k][f]), f
    assert np.array_equal(a[3]["id"], b[3]["id"])
    ca, cb = g.counters(), o.counters()
    for f in ("n_failed_step", "n_passed_step", "n_tried_step"):
        assert ca[f] == cb[f]
    ea, eb = g.events(), o.events()
    assert len(ea) == len(eb)
    for x, y in zip(ea, eb):
        for f in T.EVENT.names:
            assert x[f] == y[f], f
    return len(ea)


@pytest.mark.parametrize("n_pl", [64, 65, 95, 256, 257, 511, 513, 1024, 3071, 3072, 3073])
@pytest.mark.parametrize("n_giants", [0, 2, 3])
def test_fixed_steps(gpulib, n_pl, n_giants):
    d = bodies.make_disk(n_pl=n_pl, giants=GIANTS[:n_giants], giant_scale=(1.0,) * 3, seed=n_pl + n_giants)
    g, o = (_start(lib.System(d, bodies.thresholds()), False, 4.0) for _ in range(2))
    o.set_profiling(1)
    for s in (g, o):
        s.advance(1e9, max_steps=3)
    _same(g, o)


@pytest.mark.parametrize("n_pl,ectp", [(100, False), (400, True), (1500, False)])
def test_adaptive_steps_with_events_match_the_oracle(gpulib, n_pl, ectp):
    """A first step of 60 days is rejected; radii grown so that bodies collide and merge."""
    d = bodies.make_disk(n_pl=n_pl, giants=GIANTS[:2], seed=7, m_range=(1e-9, 1e-7))
    d.p["radius"][1:] *= 400.0
    for k in range(4):  # started next to a giant: a collision and a Hill encounter
        for f, off in zip("xyz", (0.02 + 0.03 * k, 0.01, 0.0)):
            d.r[f][10 + k] = d.r[f][1] + off
            d.v[f][10 + k] = d.v[f][1]
    thr = bodies.thresholds(ejection=30.0)
    g, o = (_start(s, True, 60.0, ectp=ectp) for s in (lib.System(d, thr), pyoracle.OracleSystem(d, thr)))
    n = 0
    for _ in range(3):
        for s in (g, o):
            s.advance(1e9, max_steps=3)
        n += _same(g, o)
    assert n > 0 and g.counters()["n_failed_step"] > 0


def test_cta_row_sum(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "cta_row_sum_gpu")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "cta_row_sum_gpu.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false", "-o", exe, src],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe, "4000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = re.findall(r"family \d warps \d+ rows \d+ bad (\d+)", r.stdout)
    assert len(rows) == 15 and all(int(b) == 0 for b in rows), r.stdout
