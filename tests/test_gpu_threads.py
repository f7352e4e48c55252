"""Contexts of different fields used by two threads at once: what one call asks
of a kernel's shared memory does not reach another's launches."""
import threading

import numpy as np
import pytest

from bqp_b200 import _native as N
from bqp_b200 import workloads

pytestmark = pytest.mark.gpu


def context(order, engine="pipeline", threads=256):
    cfg = N.default_config()
    cfg.order = order
    cfg.method = N.METHODS["dop853"]
    cfg.eps = 1e-10
    cfg.engine = N.ENGINES[engine]
    cfg.force_flags = N.FORCE_SUN
    cfg.gravity_threads = threads
    return N.Context(workloads.synthetic_field(order), cfg)


@pytest.mark.parametrize("engine,threads", [("pipeline", 256), ("pipeline", 128), ("persistent", 256)])
def test_fields_of_different_size_in_two_threads(engine, threads):
    large, small = context(70, engine, threads), context(5, engine, threads)
    x = workloads.leo_states(200, seed=3)
    want = large.propagate_final(x, workloads.EPOCH_JD, 6000.0)
    want_small = small.propagate_final(x[:20], workloads.EPOCH_JD, 600.0)
    pos = np.ascontiguousarray(x[:, :3])
    field, field_small = large.gravity(pos), small.gravity(pos)
    stop, wrong, calls = threading.Event(), [], [0]

    def small_calls():
        try:
            while not stop.is_set():
                r = small.propagate_final(x[:20], workloads.EPOCH_JD, 600.0)
                if not np.array_equal(r[0], want_small[0]):
                    wrong.append("small batch")
                if not np.array_equal(small.gravity(pos)[0], field_small[0]):
                    wrong.append("small field")
                calls[0] += 1
        except Exception as e:  # a launch refused in this thread
            wrong.append(repr(e))

    t = threading.Thread(target=small_calls)
    t.start()
    try:
        for _ in range(20):
            assert np.array_equal(large.propagate_final(x, workloads.EPOCH_JD, 6000.0)[0], want[0])
            for _ in range(20):
                assert np.array_equal(large.gravity(pos)[0], field[0])
    finally:
        stop.set()
        t.join()
    assert not wrong and calls[0] > 0
