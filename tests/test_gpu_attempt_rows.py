"""The attempt kernel's density takes its lanes, and so its order of operations,
from the rows a CTA holds on average over the launch, the same for every row: a
row's bits follow neither which rows share its CTA nor how many of those are
above ~510 km.  Rows a CTA: 28 and 34, where the rows above and below fill about
the four warps that evaluate the density; 41; 57; and its limit of 64.  Rows end
at different times, so with the exact model both lane forms run on the way.

Against the oracle at constant steps, on each side of 25 rows a CTA and at 64:
the same counts and |dr| <= 1e-9 |r|.
"""
import numpy as np
import pytest

from bqp_b200 import _native as N
from bqp_b200 import workloads
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SMS = 148


def context(atm, eps=1e-10, dt_max=300.0):
    cfg = N.default_config()
    cfg.order = 8
    cfg.method = N.METHODS["dop853"]
    cfg.eps = eps
    cfg.dt_max = dt_max
    cfg.atm_model = atm
    cfg.force_flags = N.FORCE_DRAG | N.FORCE_SUN
    return N.Context(workloads.synthetic_field(8), cfg)


def batch(n, arc):
    rng = np.random.default_rng(n)  # half of the rows below 510 km
    ang = rng.uniform(0.0, 360.0, (3, n))
    x = workloads.kep_states(workloads.RE_KM + rng.uniform(300.0, 720.0, n), rng.uniform(0.0, 0.002, n),
                             rng.uniform(0.0, 98.0, n), *ang)
    tf = np.full(n, arc)
    tf[::3] *= 0.6
    tf[1::5] *= 0.3
    return x, workloads.leo_ballistics(n, seed=1), tf


def same(a, b):
    return np.array_equal(a[0].view(np.int64), b[0].view(np.int64)) and all(np.array_equal(a[i], b[i]) for i in (1, 2, 3))


@pytest.mark.parametrize("atm", [4, 7])
@pytest.mark.parametrize("n", [28 * SMS, 5000, 6000, 57 * SMS, 64 * SMS])
def test_a_rows_bits_do_not_follow_its_neighbours(n, atm):
    ctx = context(atm)
    x, bal, tf = batch(n, 1500.0)

    def run(rows):
        return ctx.propagate_final(np.ascontiguousarray(x[rows]), workloads.EPOCH_JD, tf[rows],
                                   ballistic=np.ascontiguousarray(bal[rows]))

    order = np.arange(n)
    a = run(order)
    assert (a[1] == 0).all()
    assert same(a, run(order))
    mixed = np.random.default_rng(1).permutation(n)
    assert same([v[mixed].copy() for v in a[:4]], run(mixed))


@pytest.mark.parametrize("n,atm", [(25 * SMS, 4), (25 * SMS + 1, 4), (64 * SMS, 4), (64 * SMS, 7)])
def test_against_the_oracle(n, atm):
    x, bal, tf = batch(n, 1500.0)
    out, st, steps, evals = context(atm, eps=1e30, dt_max=30.0).propagate_final(x, workloads.EPOCH_JD, tf, ballistic=bal)
    assert (st == 0).all()
    some = np.arange(7, n, n // 40)
    F = O.Force(workloads.synthetic_field(8), 8, drag=True, sun=True, atm_model=atm)
    equ, _ = N.eci_to_equinoctial(np.ascontiguousarray(x[some]))
    d, ref_st, ref_steps, ref_evals = O.propagate_final_batch(
        F, O.ctrl("dop853", eps=1e30, dt_max=30.0), equ, workloads.EPOCH_JD, tf[some], np.ascontiguousarray(bal[some]))
    assert (ref_st == 0).all()
    assert np.array_equal(steps[some], ref_steps) and np.array_equal(evals[some], ref_evals)
    for k, i in enumerate(some):
        ref = O.equinoc2eci(equ[k], tf[i])[0] + d[k]
        assert np.linalg.norm(out[i, :3] - ref[:3]) <= 1e-9 * np.linalg.norm(ref[:3]), i
