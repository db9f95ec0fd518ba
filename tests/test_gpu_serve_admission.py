"""Admission of large networks: the reaction records a launch takes where there is
room do not keep a request out, and do not go past the budget."""
import time

import numpy as np
import pytest

from wind_b200 import lib, networks as W, serve

pytestmark = pytest.mark.gpu


def _slow(seed):
    rng = np.random.default_rng([61, seed])
    net = W.random_mass_action(rng, 4, 157, 1570, 1e-4, 1e4)
    return W.Workload(net, rng.uniform(0.0, 1.0, (4, 157)), 0.0, 1e-3, 1e-5, 1e-4)


def _bytes(wl):
    """State, network, status and step counts of a request, and its counters."""
    n = wl.net
    return wl.y0.nbytes + n.rates.nbytes + n.species.nbytes + n.nsys * 12 + 512


def test_records_do_not_narrow_admission(cuda_device):
    """Two requests of 157 species, whose records would take tens of megabytes,
    run side by side under a budget that holds their arrays only."""
    a, b = _slow(1), _slow(2)
    with serve.Server(solver="auto", hbm_budget_bytes=_bytes(a) + _bytes(b), max_inflight=4) as srv:
        deadline = time.time() + 60.0
        ia = srv.submit(a)
        while srv.stats()["running"] < 1 and time.time() < deadline:
            time.sleep(1e-4)
        ib = srv.submit(b)
        both = False
        while not both and time.time() < deadline:
            s = srv.stats()
            both = s["running"] == 2 and s["resident_bytes"] == _bytes(a) + _bytes(b)
            if s["completed"]:
                break
        assert both, s
        res = [srv.poll(i, 300.0) for i in (ia, ib)]
        assert srv.stats()["resident_bytes"] == 0
    for r, wl in zip(res, (a, b)):
        y = wl.y0.copy()
        _, st, n = lib.integrate(wl.net, y, wl.tnow, wl.tend, wl.atol, wl.rtol, "sie", "auto")
        assert np.array_equal(r.y, y) and np.array_equal(r.status, st) and np.array_equal(r.nsteps, n)


def test_records_are_counted_while_they_are_held(cuda_device):
    a = _slow(3)
    budget = 1 << 30
    with serve.Server(solver="auto", hbm_budget_bytes=budget) as srv:
        ia = srv.submit(a)
        peak = 0
        deadline = time.time() + 60.0
        while srv.stats()["completed"] == 0 and time.time() < deadline:
            peak = max(peak, srv.stats()["resident_bytes"])
        srv.poll(ia, 300.0)
        assert _bytes(a) < peak <= budget // 2
        assert srv.stats()["resident_bytes"] == 0
