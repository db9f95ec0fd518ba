"""The FP64 LU team kernel (mass action, N <= 32): every column padding at its
edges against the oracle within the plain FP64 path's 1e-10, repeated species
within a reaction, one to many teams per warp, and states, rates and pivots
that are zero or not finite beside systems that are."""
import numpy as np
import pytest

from oracle import pyoracle as O
from tests.helpers import mixed_err
from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu


def _net(n, nsys, react, lin):
    rng = np.random.default_rng([92, n, react])
    net = W.random_mass_action(rng, nsys, n, react, 1e-3, 1e2)
    if lin:
        net.linear = W.dense_linear(rng, nsys, n, 1e-2, 1e4)
    return net, rng.uniform(0.0, 1.0, (nsys, n))


@pytest.mark.parametrize("n", [1, 2, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 32])
@pytest.mark.parametrize("react_per,lin", [(10, False), (2, True), (0, True)])
def test_lu_matches_oracle(cuda_device, n, react_per, lin):
    net, y0 = _net(n, 5, react_per * n, lin)
    for ctrl in ("device", "gold"):
        y_o, y_g = y0.copy(), y0.copy()
        _, st_o, n_o = O.restated(net, y_o, 0.0, 1e-4, 1e-5, 1e-3, "sie", ctrl, threads=4)
        _, st, steps = lib.integrate(net, y_g, 0.0, 1e-4, 1e-5, 1e-3, "sie", "lu_f64", ctrl)
        assert mixed_err(y_g, y_o, 1e-5) <= 1e-10
        assert np.array_equal(st, st_o) and np.array_equal(steps, n_o)


@pytest.mark.parametrize("nsys", [1, 700, 3000, 9001])
def test_lu_teams_per_warp(cuda_device, nsys):
    """A system's result does not depend on how many share the launch."""
    net, y0 = _net(6, nsys, 30, False)
    y = y0.copy()
    _, _, n = lib.integrate(net, y, 0.0, 1e-2, 1e-6, 1e-4, "sie", "lu_f64", "gold")
    pick = np.unique(np.linspace(0, nsys - 1, 7).astype(int))
    y1 = np.ascontiguousarray(y0[pick])
    _, _, n1 = lib.integrate(net.subset(pick), y1, 0.0, 1e-2, 1e-6, 1e-4, "sie", "lu_f64", "gold")
    assert np.array_equal(y1, y[pick]) and np.array_equal(n1, n[pick])


@pytest.mark.parametrize("n", [3, 8, 16, 32])
def test_lu_nonfinite_systems_leave_the_others(cuda_device, n):
    net, y0 = _net(n, 12, 3 * n, True)
    good = [0, 5, 11]
    y0[1, 0], y0[2, n - 1], y0[3, n // 2] = np.nan, np.inf, 1e300
    net.rates[4, 0], net.rates[6, 1] = np.inf, np.nan
    net.linear[7, n - 1, n - 1] = np.inf
    net.linear[8], net.rates[8] = 0.0, 0.0   # 1 - h J_00 = 0 at h = 1: a zero pivot in column 0
    net.linear[8, 0, 0] = 1.0
    y = y0.copy()
    _, st, _ = lib.integrate(net, y, 0.0, 1.0, 1e-4, 1e-2, "sie", "lu_f64", "gold", max_attempts=400)
    y1 = np.ascontiguousarray(y0[good])
    _, st1, _ = lib.integrate(net.subset(np.array(good)), y1, 0.0, 1.0, 1e-4, 1e-2, "sie", "lu_f64", "gold",
                              max_attempts=400)
    assert np.array_equal(y[good], y1) and np.array_equal(st[good], st1)
    for s in (1, 2, 4, 6, 7):
        assert st[s] & 1 and not np.isfinite(y[s]).all()
