"""The CTA kernel's MIXED solve at the edges of its panels, tiles and thread
counts, against the FP64 oracle within the mixed path's 1e-5: whole and ragged
panels, the pivoted inverse, reaction records in shared memory and in global
scratch, and networks whose lists do not fit the records (a species in every
reaction, a launch without scratch)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from tests.helpers import mixed_err
from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu


def _net(n, nsys, react, k=(1e-3, 1e3)):
    rng = np.random.default_rng([93, n, react])
    return W.random_mass_action(rng, nsys, n, react, *k), rng.uniform(0.0, 1.0, (nsys, n))


def _check(net, y0, dt, ctrl="gold", attempts=24):
    y_o, y_g = y0.copy(), y0.copy()
    O.restated(net, y_o, 0.0, dt, 1e-4, 1e-3, "sie", ctrl, max_attempts=attempts, threads=4)
    _, st, _ = lib.integrate(net, y_g, 0.0, dt, 1e-4, 1e-3, "sie", "mixed", ctrl, max_attempts=attempts)
    assert mixed_err(y_g, y_o, 1e-4) <= 1e-5
    return st


@pytest.mark.parametrize("n", [33, 47, 48, 49, 64, 95, 96, 97, 112, 127, 128, 129, 144, 157, 160, 176])
def test_cta_mixed_edges(cuda_device, n):
    net, y0 = _net(n, 3, 10 * n)
    _check(net, y0, 1e-4)


@pytest.mark.parametrize("n,react", [(40, 400), (64, 640), (157, 700)])
def test_cta_mixed_hub_species(cuda_device, n, react):
    """Species 0 takes part in every reaction: its list is longer than the
    records have room for."""
    net, y0 = _net(n, 3, react, (1e-3, 1e1))
    net.species[:, :, 0] = 0
    _check(net, y0, 1e-4)


@pytest.mark.parametrize("n", [48, 100, 157])
def test_cta_mixed_large_steps(cuda_device, n):
    """Steps at which the unpivoted inverse fails (flag REFINE_FALLBACK) end at
    the FP64 LU's result."""
    net, y0 = _net(n, 4, 6 * n, (1e-2, 1e4))
    y_l, y_g = y0.copy(), y0.copy()
    lib.integrate(net, y_l, 0.0, 1.0, 1e-3, 1e-2, "sie", "lu_f64", "gold")
    _, st, _ = lib.integrate(net, y_g, 0.0, 1.0, 1e-3, 1e-2, "sie", "mixed", "gold")
    assert (st & 8).any()
    assert mixed_err(y_g, y_l, 1e-3) <= 1e-5


@pytest.mark.parametrize("solver,n", [("mixed", 157), ("lu_f64", 128)])
def test_cta_launch_without_scratch(cuda_device, solver, n):
    """Networks whose records do not fit shared memory, through the entry point
    that allocates nothing (species lists) and the one that does (records in
    scratch): the same terms in the same order, so the same bits."""
    net, y0 = _net(n, 3, 10 * n)
    wl = [W.Workload(net, y0, 0.0, 1e-5, 1e-4, 1e-3)]
    (want, st, steps), = lib.integrate_batch(wl, "sie", solver, "gold")
    (got, s, c), = lib.integrate_batch(wl, "sie", solver, "gold", noalloc=True)
    assert steps.min() > 0
    assert np.array_equal(got, want) and np.array_equal(s, st) and np.array_equal(c, steps)
