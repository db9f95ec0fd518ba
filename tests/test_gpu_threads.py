"""Host threads that integrate at the same time.  Batches of one network but of
different sizes put different numbers of teams into a block, hence different
shared-memory sizes of one kernel: no thread's launch may be refused because of
another's, and every result is that of the call made alone."""
import threading

import numpy as np
import pytest

from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["lu_f64", "gje_f64", "mixed"])
def test_threads_with_batches_of_different_sizes(cuda_device, solver):
    n, sizes, calls = 5, (8, 2000, 9000), 150
    rng = np.random.default_rng(41)
    jobs = []
    for k, nsys in enumerate(sizes):
        # (mixed: the block's size depends on the reactions only)
        net = W.random_mass_action(rng, nsys, n, 10 + (40 * k if solver == "mixed" else 0), 1e-3, 1e1)
        y0 = rng.uniform(0.0, 1.0, (nsys, n))
        want = y0.copy()
        _, st, steps = lib.integrate(net, want, 0.0, 1e-3, 1e-2, 1e-2, "sie", solver, max_attempts=2)
        jobs.append((net, y0, want, st, steps))
    wrong = []

    def work(net, y0, want, st, steps):
        try:
            for _ in range(calls):
                y = y0.copy()
                _, s, c = lib.integrate(net, y, 0.0, 1e-3, 1e-2, 1e-2, "sie", solver, max_attempts=2)
                if not (np.array_equal(y, want) and np.array_equal(s, st) and np.array_equal(c, steps)):
                    raise AssertionError("a result differs from the call made alone")
        except Exception as e:
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
