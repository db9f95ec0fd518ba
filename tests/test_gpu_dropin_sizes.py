"""The drop-in's float32 call around the size up to which the arrays and the
total travel in one copy each: the oracle on the same inputs, rounded back."""
import numpy as np
import pytest

from oracle import pyoracle as O
from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsys", [1, 545, 546, 547, 3001])
def test_dropin_packed_and_plain_copies(cuda_device, nsys):
    wl = W.workload_katz96(nsys, seed=61)
    f32 = np.float32
    c32 = np.ascontiguousarray(wl.net.constants.astype(f32))
    y32 = np.ascontiguousarray(wl.y0.astype(f32))
    y_o = y32.astype(np.float64)
    net64 = W.Network(wl.net.kind, 5, nsys, constants=c32.astype(np.float64))
    tot, _, _ = O.restated(net64, y_o, 0.0, float(f32(1e10)), float(f32(5e-3)), float(f32(5e-3)), "sie", "device",
                           threads=4)
    n = lib.legacy("katz96", "sie")(f32(0.0), f32(1e10), 1, c32.ctypes.data, y32.ctypes.data, nsys, 5, f32(5e-3),
                                    f32(5e-3))
    assert np.array_equal(y32, y_o.astype(f32)) and n == tot
