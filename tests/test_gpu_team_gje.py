"""The team kernel's Gauss-Jordan by columns against the oracle's full-width
elimination, bit for bit: team sizes 8/16/32 at their edges, repeated species
within a reaction, one to many teams per warp, and pivots or states that are
zero or not finite (the full-width path)."""
import numpy as np
import pytest

from oracle import pyoracle as O
from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu


def _net(n, nsys, react, lin):
    rng = np.random.default_rng([91, n, react])
    net = W.random_mass_action(rng, nsys, n, react, 1e-3, 1e3)
    if lin:
        net.linear = W.dense_linear(rng, nsys, n, 1e-2, 1e4)
    return net, rng.uniform(0.0, 1.0, (nsys, n))


def _check(net, y0, dt, ctrl, method="sie", attempts=40):
    y_o, y_g = y0.copy(), y0.copy()
    tot_o, st_o, n_o = O.restated(net, y_o, 0.0, dt, 1e-6, 1e-4, method, ctrl, max_attempts=attempts, threads=4)
    tot, st, n = lib.integrate(net, y_g, 0.0, dt, 1e-6, 1e-4, method, "gje_f64", ctrl, max_attempts=attempts)
    assert np.array_equal(y_g, y_o, equal_nan=True)
    assert tot == tot_o and np.array_equal(n, n_o) and np.array_equal(st, st_o)


@pytest.mark.parametrize("ctrl", ["device", "gold"])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32])
def test_team_gje_matches_oracle(cuda_device, n, ctrl):
    for react, lin in ((10 * n, False), (3, True)):
        net, y0 = _net(n, 5, react, lin)
        _check(net, y0, 1e-3, ctrl)
    _check(net, y0, 1e-3, ctrl, "rk2")


@pytest.mark.parametrize("nsys", [1, 600, 2500, 9001])
def test_team_gje_teams_per_warp(cuda_device, nsys):
    net, y0 = _net(5, nsys, 20, False)
    _check(net, y0, 1e-3, "gold", attempts=12)


@pytest.mark.parametrize("n", [3, 8, 16, 32])
def test_team_gje_zero_pivot_and_nonfinite(cuda_device, n):
    net, y0 = _net(n, 8, 2 * n, True)
    net.linear[0] = 0.0
    net.linear[0, 0, 0] = 1.0        # 1 - h J_00 = 0 at h = 1
    net.rates[0] = 0.0
    net.linear[1, n - 1, n - 1] = np.inf
    y0[2, 0], y0[3, n - 1], y0[4, 0], y0[5, 1 % n] = np.nan, np.inf, 1e300, -0.0
    net.rates[6, 0] = np.inf
    _check(net, y0, 1.0, "device", attempts=20)
    _check(net, y0, 1.0, "gold", attempts=20)
