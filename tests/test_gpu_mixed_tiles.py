"""The packed mixed kernel at the edges of its sink pairs, warps' slices, source tiles and
source chunks.

Tolerance: a light pair's FP32 term has fewer than 16 roundings of at most 2**-24 (the
displacement and the squared distance 5, rsqrt.approx and its correction 4, the mass and the
products 4), so a body's acceleration is off by about 2**-20 of the sum of its light terms'
sizes at most (a slice's 32 terms round the sum either way); the heavy terms and the two-sum accumulation add less than 2**-42 of the whole.
"""
import numpy as np
import pytest

from redgb import bodies, lib, types as T

pytestmark = pytest.mark.gpu


def light_sizes(disk):
    """Per body, the sum over the light bodies of m / r**2 (float64; G = 1 in the code's units)."""
    r = np.stack([disk.r[f] for f in "xyz"], 1)
    m = np.where(np.arange(disk.n_total) == 0, 0.0, disk.p["mass"])
    d2 = ((r[:, None] - r[None]) ** 2).sum(-1)
    np.fill_diagonal(d2, np.inf)
    return (m[None] / d2).sum(1)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 65, 126, 127, 128, 129, 255, 256, 257, 511, 513, 1300])
def test_mixed_tile_edges(gpulib, n):
    disk = bodies.make_disk(n_pl=n, pl_type=T.BODY_PROTOPLANET, giants=(), seed=n)
    g = lib.System(disk, bodies.thresholds())
    ref = g.calc_accel()
    a_e = np.stack([ref[f] for f in "xyz"], 1)
    tol = 2.0 ** -20 * light_sizes(disk) + 2.0 ** -42 * np.linalg.norm(a_e, axis=1)
    g.set_gravity_mode(T.GRAVITY_MIXED)
    for chunk in (0, 256, 512):  # the rule's, one tile, two tiles per chunk
        g.set_launch_shape(mixed_chunks=chunk)
        am = g.calc_accel()
        err = np.linalg.norm(np.stack([am[f] for f in "xyz"], 1) - a_e, axis=1)
        assert (err <= tol).all(), (n, chunk, float((err / tol).max()))


@pytest.mark.parametrize("n_emb,n_pl,n_tp", [(70, 1, 1), (100, 129, 0), (130, 0, 300), (300, 700, 257)])
def test_blocks_in_one_launch(gpulib, n_emb, n_pl, n_tp):
    """The three interaction blocks' tiles in one launch, each block with its own source count
    and chunks."""
    rng = np.random.RandomState(n_emb)
    emb = [(10.0 ** rng.uniform(-9, -7), 1.0 + 3.0 * k / n_emb, 0.02) for k in range(n_emb)]
    disk = bodies.make_disk(n_pl=n_pl, embryos=emb, giants=((9.55e-4, 5.2, 0.05),), n_tp=n_tp, seed=n_pl)
    g = lib.System(disk, bodies.thresholds())
    ref = g.calc_accel()
    a_e = np.stack([ref[f] for f in "xyz"], 1)
    m = disk.p["mass"].copy()
    m[:2] = 0.0
    r = np.stack([disk.r[f] for f in "xyz"], 1)
    d2 = ((r[:, None] - r[None]) ** 2).sum(-1)
    np.fill_diagonal(d2, np.inf)
    tol = 2.0 ** -20 * (m[None] / d2).sum(1) + 2.0 ** -42 * np.linalg.norm(a_e, axis=1)
    g.set_gravity_mode(T.GRAVITY_MIXED)
    for chunk in (0, 256, 512):
        g.set_launch_shape(mixed_chunks=chunk)
        am = g.calc_accel()
        err = np.linalg.norm(np.stack([am[f] for f in "xyz"], 1) - a_e, axis=1)
        assert (err <= tol).all(), (chunk, float((err / tol).max()))
