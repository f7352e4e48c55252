"""The attempt kernel at the largest fields whose table it holds beside its sums:
order 82 (83 and up run in the stage kernels) and, for sigma points with their
larger table of cells, order 76 (77 and up).

Against the oracle at constant steps: the same counts and |dr| <= 1e-9 |r|.
Sigma points take the same bits in both engines' kernels (runs timed by kernel
class are the stage kernels').
"""
import numpy as np
import pytest

from bqp_b200 import _native as N
from bqp_b200 import workloads
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def context(order, atm, **kw):
    cfg = N.default_config()
    cfg.order = order
    cfg.method = N.METHODS["dop853"]
    cfg.atm_model = atm or 4
    cfg.force_flags = N.FORCE_SUN | (N.FORCE_DRAG if atm else 0)
    for k, v in kw.items():
        setattr(cfg, k, v)
    return N.Context(workloads.synthetic_field(order), cfg)


@pytest.mark.parametrize("atm", [0, 7])
@pytest.mark.parametrize("order", [82, 83])
def test_against_the_oracle(order, atm):
    n = 150
    x = workloads.leo_states(n, seed=order)
    bal = workloads.leo_ballistics(n, seed=1)
    out, st, steps, evals = context(order, atm, eps=1e30, dt_max=30.0).propagate_final(
        x, workloads.EPOCH_JD, 600.0, ballistic=bal)
    assert (st == 0).all()
    some = np.arange(0, n, 15)
    F = O.Force(workloads.synthetic_field(order), order, drag=bool(atm), sun=True, atm_model=atm or 4)
    equ, _ = N.eci_to_equinoctial(np.ascontiguousarray(x[some]))
    d, ref_st, ref_steps, ref_evals = O.propagate_final_batch(
        F, O.ctrl("dop853", eps=1e30, dt_max=30.0), equ, workloads.EPOCH_JD, 600.0, np.ascontiguousarray(bal[some]))
    assert (ref_st == 0).all()
    assert np.array_equal(steps[some], ref_steps) and np.array_equal(evals[some], ref_evals)
    for k, i in enumerate(some):
        ref = O.equinoc2eci(equ[k], 600.0)[0] + d[k]
        assert np.linalg.norm(out[i, :3] - ref[:3]) <= 1e-9 * np.linalg.norm(ref[:3]), i


@pytest.mark.parametrize("order", [76, 77])
def test_sigma_points_take_the_same_bits(order):
    mean, cov = workloads.ukf_objects(90, seed=4)
    ctx = context(order, 4, eps=1e-10)
    a = ctx.sigma_propagate(mean, cov, workloads.EPOCH_JD, 1500.0)
    ctx.profile(True)
    b = ctx.sigma_propagate(mean, cov, workloads.EPOCH_JD, 1500.0)
    assert (a[2] == 0).all()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and np.array_equal(a[3], b[3])
