"""Teams of up to 32 species with many reactions: the lists a system is staged
into (whole and partial words of 32 reactions, a species in every reaction,
catalysts), the Jacobian summed in place where the sorted terms would leave one
team per SM, and what staging costs beside an attempt."""
import time

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.helpers import mixed_err
from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu


def _net(n, nsys, react, seed, k=(1e-3, 1e1)):
    rng = np.random.default_rng([seed, n, react])
    net = W.random_mass_action(rng, nsys, n, react, *k)
    if react >= 4:
        net.species[:, 0] = [0, 0, 0, n - 1]   # 2 A -> A + B
        net.species[:, 1] = [n - 1, 0, n - 1, 0]  # nothing changes
        net.species[:, 2] = [0, 0, n - 1, n - 1]
        net.species[:, react - 1, 0] = 0
    return net, rng.uniform(0.0, 1.0, (nsys, n))


@pytest.mark.parametrize("react", [1, 31, 32, 33, 64, 65, 200])
@pytest.mark.parametrize("n", [1, 3, 8, 16, 32])
def test_lists_around_a_word(cuda_device, n, react):
    net, y0 = _net(n, 4, react, 7)
    if n == 8:
        net.species[:, :, 1] = 2  # in every reaction
    for method in ("sie", "rk2"):
        y_o, y_g = y0.copy(), y0.copy()
        _, _, n_o = O.restated(net, y_o, 0.0, 1e-3, 1e-4, 1e-3, method, "gold", max_attempts=12, threads=4)
        _, _, n_g = lib.integrate(net, y_g, 0.0, 1e-3, 1e-4, 1e-3, method, "gje_f64", "gold", max_attempts=12)
        assert np.array_equal(y_g, y_o) and np.array_equal(n_g, n_o)
    y_o, y_l = y0.copy(), y0.copy()
    O.restated(net, y_o, 0.0, 1e-4, 1e-5, 1e-3, "sie", "gold", threads=4)
    lib.integrate(net, y_l, 0.0, 1e-4, 1e-5, 1e-3, "sie", "lu_f64", "gold")
    assert mixed_err(y_l, y_o, 1e-5) <= 1e-10  # the plain FP64 path's bound


@pytest.mark.parametrize("n,react", [(17, 1800), (24, 1800), (32, 1700), (32, 1900)])
def test_jacobian_in_place(cuda_device, n, react):
    """More systems than SMs take the in-place Jacobian, the same ones in parts
    the sorted terms: the same bits."""
    import torch
    nsys = torch.cuda.get_device_properties(cuda_device).multi_processor_count + 2
    net, y0 = _net(n, nsys, react, 8, (1e-4, 1e2))
    net.species[:, : react // 4, 2] = 1
    whole = y0.copy()
    _, st, steps = lib.integrate(net, whole, 0.0, 1e-4, 1e-6, 1e-5, "sie", "lu_f64", "device", max_attempts=8)
    for part in (slice(0, nsys // 2), slice(nsys // 2, nsys)):
        w = W.Workload(net, y0, 0.0, 1e-4, 1e-6, 1e-5).subset(part)
        y = np.ascontiguousarray(w.y0).copy()
        _, s, c = lib.integrate(w.net, y, 0.0, 1e-4, 1e-6, 1e-5, "sie", "lu_f64", "device", max_attempts=8)
        assert np.array_equal(y, whole[part])
        assert np.array_equal(s, st[part]) and np.array_equal(c, steps[part])


def test_staging_does_not_outweigh_an_attempt(cuda_device):
    """One attempt of 2,000 systems with 1,900 reactions: the LU team, whose lists
    are the longer ones, within three times the MIXED team."""
    import torch
    n, react, nsys = 32, 1900, 2000
    few, y = _net(n, 50, react, 9)
    rep = nsys // 50
    arrays = {"rates": torch.from_numpy(np.tile(few.rates, (rep, 1))).cuda(),
              "species": torch.from_numpy(np.tile(few.species, (rep, 1, 1))).cuda()}
    net = W.Network(W.NET_MASS_ACTION, n, nsys, rates=np.tile(few.rates, (rep, 1)),
                    species=np.tile(few.species, (rep, 1, 1)))
    y0 = torch.from_numpy(np.tile(y, (rep, 1))).cuda()
    best = {}
    for solver in ("lu_f64", "mixed"):
        for _ in range(5):
            yd = y0.clone()
            torch.cuda.synchronize()
            t = time.perf_counter()
            lib.integrate(net, yd, 0.0, 1e-5, 1e-6, 1e-6, "sie", solver, "device", max_attempts=1,
                          device_arrays=arrays)
            best[solver] = min(best.get(solver, 1e9), time.perf_counter() - t)
    assert best["lu_f64"] <= 3.0 * best["mixed"], best


@pytest.mark.parametrize("solver", ["auto", "gje_f64"])
@pytest.mark.parametrize("n,react", [(16, 300), (16, 301), (32, 384), (32, 385)])
def test_batch_staging_on_both_sides_of_the_rule(cuda_device, n, react, solver):
    """A group's result in a batch, staged either way, is the one of the call of
    its own: bit for bit for Gauss-Jordan, within the plain FP64 path's bound for
    the LU."""
    net, y0 = _net(n, 6, react, 10)
    alone = y0.copy()
    _, st, steps = lib.integrate(net, alone, 0.0, 1e-4, 1e-5, 1e-3, "sie", solver, "gold")
    (y, s, c), = lib.integrate_batch([W.Workload(net, y0, 0.0, 1e-4, 1e-5, 1e-3)], "sie", solver, "gold")
    assert np.array_equal(s, st) and np.array_equal(c, steps)
    if solver == "gje_f64":
        assert np.array_equal(y, alone)
    else:
        assert mixed_err(y, alone, 1e-5) <= 1e-10
