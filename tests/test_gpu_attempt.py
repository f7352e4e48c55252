"""The attempt kernel (a whole step attempt of a small batch in one launch)
against the stage kernels, at the sizes where it changes: one row, one and two
rows a CTA, one and two tiles of a warp, its last size and the first it leaves
to the stage kernels.  A gravity_threads other than the default keeps a batch
on the stage kernels.

Tolerance: two adaptive solutions of the same equations, each within
10 eps a step of the exact one (as the engines' comparison with the oracle),
which holds where the force is smooth on the scale of a step.  Without the
field (order 0) steps grow to dt_max and JB2008's branches in altitude (its
local-time correction ends at 800 km) set the difference of any two solutions,
so that case is checked where the rows take the same bits: sigma points.
"""
import numpy as np
import pytest

from bqp_b200 import _native as N
from bqp_b200 import workloads

pytestmark = pytest.mark.gpu

EPS = 1e-10
SMS = 148


def context(order, method, atm, flags, frame="gmst", stages=False, fp32=False):
    cfg = N.default_config()
    cfg.order = order
    cfg.method = N.METHODS[method]
    cfg.eps = EPS
    cfg.atm_model = atm
    cfg.force_flags = flags | (N.FORCE_DRAG if atm else 0)
    cfg.drag_fp32 = int(fp32)
    cfg.gravity_threads = 128 if stages else 256
    ctx = N.Context(workloads.synthetic_field(max(order, 2)), cfg)
    if frame != "gmst":
        ctx.set_frame(frame)
    return ctx


@pytest.mark.parametrize("n,order,method,atm,flags,frame,arc,fp32", [
    (1, 5, "vern7", 7, 4 | 8, "iau2006", 4000.0, False),
    (SMS + 1, 20, "dop853", 4, 4, "gmst", 1500.0, False),
    (32 * SMS, 3, "dopri5", 0, 8, "gmst", 600.0, False),
    (32 * SMS + 1, 8, "vern9", 5, 0, "iau2006", 600.0, False),
    (64 * SMS, 6, "dopri5_solver", 6, 4, "gmst", 300.0, True),
    (64 * SMS + 1, 6, "vern7", 7, 4, "gmst", 300.0, False),
    (300, 78, "dop853", 4, 4 | 8, "iau2006", 600.0, False),
    (65, 12, "vern7", 7, 2 | 4 | 8, "iau2006", 6000.0, False),
])
def test_attempt_kernel_against_the_stage_kernels(n, order, method, atm, flags, frame, arc, fp32):
    x = workloads.leo_states(n, seed=n)
    bal = workloads.leo_ballistics(n, seed=1)
    tf = np.full(n, arc)
    tf[::3] *= 0.6  # rows that end earlier
    a = context(order, method, atm, flags, frame, fp32=fp32).propagate_final(x, workloads.EPOCH_JD, tf, ballistic=bal)
    b = context(order, method, atm, flags, frame, True, fp32).propagate_final(x, workloads.EPOCH_JD, tf, ballistic=bal)
    assert np.array_equal(a[1], b[1]) and (a[1] == 0).all()
    dr = np.linalg.norm(a[0][:, :3] - b[0][:, :3], axis=1)
    bound = 2 * 10 * EPS * np.maximum(np.maximum(a[2], b[2]), 10)
    if fp32:  # the FP32 density's rounding, 1e-5 of the drag displacement
        bound = bound + 1e-5 * 1e-9 * tf ** 2
    assert (dr <= bound).all(), (dr / bound).max()


def test_sampled_rows_and_failures():
    n = 40
    x = workloads.leo_states(n, seed=9)
    x[3] = np.nan
    x[17, 3:] *= 2.0  # unbound
    grid = np.arange(0.0, 3001.0, 150.0)
    r = [context(20, "dop853", 7, 4 | 8, "iau2006", s).propagate_sampled(x, workloads.EPOCH_JD, 3000.0, grid)
         for s in (False, True)]
    assert np.array_equal(r[0][1], r[1][1])
    assert r[0][1][3] == 3 and r[0][1][17] == 3 and np.isnan(r[0][0][[3, 17]]).all()
    ok = r[0][1] == 0
    assert ok.sum() == n - 2
    dr = np.linalg.norm(r[0][0][ok, :, :3] - r[1][0][ok, :, :3], axis=2)
    assert dr.max() <= 2e-5  # interior samples: the Hermite interpolant's own error


@pytest.mark.parametrize("order,atm,frame", [(20, 0, "gmst"), (20, 4, "gmst"), (20, 7, "gmst"), (20, 4, "iau2006"),
                                             (20, 7, "iau2006"), (0, 4, "gmst"), (0, 7, "iau2006")])
def test_sigma_points_take_the_same_bits(order, atm, frame):
    """Kernels timed by class run as stage kernels; the rows keep their order
    of operations in both."""
    mean, cov = workloads.ukf_objects(90, seed=4)
    ctx = context(order, "dop853", atm, 4 | 8, frame)
    a = ctx.sigma_propagate(mean, cov, workloads.EPOCH_JD, 3000.0)
    ctx.profile(True)
    b = ctx.sigma_propagate(mean, cov, workloads.EPOCH_JD, 3000.0)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and np.array_equal(a[3], b[3])
