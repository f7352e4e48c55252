"""The wall-clock limit of a call (max_kernel_seconds) that runs out: rows that
have not finished end with the watchdog's status, at most eight attempts after
it in the stage-synchronous engine's kernels -- the stage kernels look at the
clock after every two attempts with two more in flight, the attempt kernel
after each --, and rows that four attempts finish are finished.  The limit here
is over before the first attempt ends.
"""
import numpy as np
import pytest

from bqp_b200 import _native as N
from bqp_b200 import workloads

pytestmark = pytest.mark.gpu

ATTEMPTS = 8


def context(threads=256, flags=0, limit=1e-6):
    cfg = N.default_config()
    cfg.order = 20
    cfg.method = N.METHODS["dop853"]
    cfg.eps = 1e-10
    cfg.atm_model = 7
    cfg.cr = 1.3
    cfg.force_flags = flags
    cfg.max_kernel_seconds = limit
    cfg.gravity_threads = threads
    return N.Context(workloads.synthetic_field(20), cfg)


@pytest.mark.parametrize("n,threads,flags", [
    (1, 256, 0), (300, 256, N.FORCE_DRAG | N.FORCE_SUN), (300, 256, N.FORCE_SUN | N.FORCE_SRP),
    (300, 128, N.FORCE_DRAG), (9473, 256, N.FORCE_DRAG)])
def test_final_rows(n, threads, flags):
    x = workloads.leo_states(n, seed=2)
    tf = np.full(n, 86400.0)
    tf[1::4] = 0.5  # one step's worth
    out, st, steps, evals = context(threads, flags).propagate_final(x, workloads.EPOCH_JD, tf)
    long = tf > 1.0
    assert (st[long] == 10).all() and np.isnan(out[long]).all()
    assert (st[~long] == 0).all() and np.isfinite(out[~long]).all()
    assert steps.max() <= ATTEMPTS
    assert evals.max() <= 13 * ATTEMPTS  # twelve stages and, with SRP, the dense one


def test_sigma_points():
    mean, cov = workloads.ukf_objects(20, seed=4)
    r = context(flags=N.FORCE_SUN).sigma_propagate(mean, cov, workloads.EPOCH_JD, 86400.0)
    assert np.isnan(r[0]).all() and (r[2] == 10).all()
    assert r[3].max() <= 7 * 12 * ATTEMPTS


def test_a_limit_that_is_not_reached_changes_nothing():
    x = workloads.leo_states(300, seed=5)
    a = context(limit=3600.0).propagate_final(x, workloads.EPOCH_JD, 3000.0)
    b = context(limit=60.0).propagate_final(x, workloads.EPOCH_JD, 3000.0)
    assert (a[1] == 0).all() and np.array_equal(a[0].view(np.int64), b[0].view(np.int64))
