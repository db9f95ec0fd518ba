"""The refinement of the CTA kernel's MIXED solve after a pivoted inverse.

f = L y, L skew but for L_00 = 2: at h/2 = 1/2 the first diagonal element of
A = I - (h/2) L is exactly zero, so the unpivoted FP32 inverse is not finite and
the pivoted one, whose last pivot is far above |x|, is refined.  One attempt at
a tolerance that accepts it ends at the two half steps y + (h/2) A^-1 L y, here
from numpy in FP64.

Tolerance: a refinement ends at a predicted error of 2^-33 max|x| with a
contraction of at most 1/2, so its error is below 2^-32 max|x|; rounding of the
FP64 residual adds N 2^-52 times the condition number of A; the second half step
turns an error e of the first into A^-1 e."""
import numpy as np
import pytest

from wind_b200 import lib, networks as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [63, 64, 65, 127, 157])
def test_pivoted_inverse_is_refined_against_the_solution(cuda_device, n):
    rng = np.random.default_rng([17, n])
    nsys, h = 96, 1.0
    g = rng.standard_normal((nsys, n, n))
    lin = g - np.swapaxes(g, 1, 2)
    lin *= (10.0 ** rng.uniform(2.5, 4.0, nsys) / np.linalg.norm(lin, 2, (1, 2)))[:, None, None]
    lin[:, 0, 0] = 2.0
    lin = lin.astype(np.float32)
    y0 = rng.uniform(-1.0, 1.0, (nsys, n))
    net = W.Network(W.NET_MASS_ACTION, n, nsys, linear=lin)
    y = y0.copy()
    _, st, steps = lib.integrate(net, y, 0.0, h, 1e30, 1e30, "sie", "mixed", "gold")
    assert (steps == 3).all()
    assert (st & 8).all()  # REFINE_FALLBACK: the pivoted inverse ran
    m = lin.astype(np.float64)
    a = np.eye(n) - 0.5 * h * m
    inv_norm = np.abs(np.linalg.inv(a)).sum(2).max(1)
    cond = inv_norm * np.abs(a).sum(2).max(1)
    want, xmax = y0.copy(), []
    for _ in range(2):
        x = np.linalg.solve(a, np.einsum("sij,sj->si", m, want)[..., None])[..., 0]
        want = want + 0.5 * h * x
        xmax.append(np.abs(x).max(1))
    tol = 0.5 * h * (2.0 ** -32 + n * 2.0 ** -52 * cond) * (xmax[1] + inv_norm * xmax[0])
    err = np.abs(y - want).max(1)
    assert (err <= tol).all(), (int((err > tol).sum()), float((err / tol).max()))
