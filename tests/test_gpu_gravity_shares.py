"""The gravity kernels' splits -- rows a lane, warps to a tile, CTAs to a
cluster -- against the oracle, at the sizes where a split changes: tiles of
32 x 1..4 rows, one more and one less, the clusters' row limits, the orders at
which the table needs two and three CTAs, the smallest order and the oracle's largest.

Tolerance: the force call's, |da| <= 1e-12 |a| with the point mass included.
"""
import numpy as np
import pytest

from bqp_b200 import _native as N
from bqp_b200 import workloads
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def positions(n, seed):
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(n, 3))
    u *= (rng.uniform(6578.0, 42164.0, n) / np.linalg.norm(u, axis=1))[:, None]
    # the polar axis and the equator: powers of x + i y and z that vanish
    u[0] = (0.0, 0.0, 6800.0)
    u[-1] = (6800.0, 0.0, 0.0)
    return u


def context(order, threads=256, slots=4):
    cfg = N.default_config()
    cfg.order = order
    cfg.gravity_threads, cfg.gravity_slots = threads, slots
    return N.Context(workloads.synthetic_field(order), cfg)


def check(ctx, order, n, seed):
    pos = positions(n, seed)
    acc, st = ctx.gravity(pos)
    assert (st == 0).all()
    some = np.unique(np.concatenate([[0, n - 1], np.random.default_rng(seed).integers(0, n, 40)]))
    F = O.Force(workloads.synthetic_field(order), order, drag=False, sun=False, moon=False)
    ref = F.gravity_itrs(pos[some])
    err = np.linalg.norm(acc[some] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() <= 1e-12, (order, n, err.max())
    assert np.isfinite(acc).all()
    return pos, acc


@pytest.mark.parametrize("order", [2, 3, 39, 40, 59, 60, 70, 78, 79, 104, 105, 120])
def test_sizes_around_the_splits(order):
    ctx = context(order)
    for n in (1, 2, 31, 33, 129, 1500, 1501, 3000, 3001, 9473):
        check(ctx, order, n, seed=n + order)


@pytest.mark.parametrize("threads,slots", [(32, 1), (64, 4), (96, 2), (160, 4), (256, 1), (256, 2)])
def test_configured_threads_and_rows(threads, slots):
    ctx = context(70, threads, slots)
    for n in (5, 700, 20011):
        check(ctx, 70, n, seed=n)


def test_invalid_rows_among_valid_ones_in_a_cluster():
    ctx = context(70)
    pos = positions(900, 3)
    bad = [0, 31, 32, 127, 500, 899]
    good, _ = ctx.gravity(pos)
    pos[bad] = [[np.nan, 0, 0], [0, 0, 0], [np.inf, 1, 1], [0, 0, 0], [np.nan] * 3, [0, 0, 0]]
    acc, st = ctx.gravity(pos)
    rest = np.setdiff1d(np.arange(900), bad)
    assert (st[bad] == N.ST_GRAVITY_RADIUS).all() and np.isnan(acc[bad]).all()
    assert (st[rest] == 0).all() and np.array_equal(acc[rest], good[rest])
