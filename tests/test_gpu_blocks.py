"""The compiled networks' block solvers: the Gauss-Jordan inverse by diagonal
blocks against the oracle's full-width elimination, bit for bit, including
states and constants that are zero, huge or not finite (where the full-width
elimination spreads infinities and NaN across blocks), and the block LU
against the oracle within the plain FP64 path's 1e-10."""
import numpy as np
import pytest

from oracle import pyoracle as O
from tests.helpers import mixed_err
from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu

VALUES = [0.0, -0.0, np.nan, np.inf, -np.inf, 1e300, -1e300, 1e-310]


def _cases(net):
    if net == "katz96":
        wl = W.workload_katz96(48, seed=51)
        return wl.net, wl.y0.copy(), 1e10
    if net == "nr":
        wl = W.workload_nr(48, seed=52)
        return wl.net, wl.y0.copy(), 0.01
    return W.stifftrig(48), np.tile([0.0, 1.0], (48, 1)).astype(np.float64), 0.25


@pytest.mark.parametrize("ctrl", ["device", "gold"])
@pytest.mark.parametrize("net", ["katz96", "nr", "trig"])
def test_block_gje_special_values(cuda_device, net, ctrl):
    nw, y0, dt = _cases(net)
    nw.constants = nw.constants.copy()
    N, NC = y0.shape[1], nw.constants.shape[1]
    for i, v in enumerate(VALUES):
        for e in range(min(N, 2)):
            y0[2 * i + e, (i + 3 * e) % N] = v
        nw.constants[16 + 2 * i, i % NC] = v
        nw.constants[17 + 2 * i, (i + NC // 2) % NC] = v
    nw.constants[40] = 1.0 / dt    # pivots 1 - h J that cancel
    nw.constants[41] = -1.0 / dt
    y_o, y_g = y0.copy(), y0.copy()
    _, st_o, n_o = O.restated(nw, y_o, 0.0, dt, 1e-6, 1e-4, "sie", ctrl, max_attempts=60, threads=4)
    _, st, n = lib.integrate(nw, y_g, 0.0, dt, 1e-6, 1e-4, "sie", "gje_f64", ctrl, max_attempts=60)
    assert np.array_equal(y_g, y_o, equal_nan=True)
    assert np.array_equal(n, n_o) and np.array_equal(st, st_o)


@pytest.mark.parametrize("net", ["katz96", "nr", "trig"])
def test_block_lu_matches_oracle(cuda_device, net):
    nw, y0, dt = _cases(net)
    y_o, y_g = y0.copy(), y0.copy()
    O.restated(nw, y_o, 0.0, dt, 1e-8, 1e-6, "sie", "gold", threads=4)
    lib.integrate(nw, y_g, 0.0, dt, 1e-8, 1e-6, "sie", "lu_f64", "gold")
    assert mixed_err(y_g, y_o, 1e-8) <= 1e-10
