"""The CTA kernel's block size (cta_block_threads in wind_b200/csrc/cta_kernel.cuh):
every block has a thread per equation, half blocks only go where they are the
faster ones, and a system's result does not depend on the choice."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from wind_b200 import _capi, lib, networks as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include "cta_kernel.cuh"
using namespace wind;
int main() {
    for (int n = 33; n <= CTA_MAXN; n++)
        for (int solver = 0; solver < 3; solver++)
            for (int many = 0; many < 2; many++)
                printf("%d %d %d %d %d %d\n", n, solver, many, cta_block_threads(n, solver, false, false, many != 0),
                       cta_block_threads(n, WIND_SOLVER_LU_F64, true, false, many != 0),
                       cta_block_threads(n, WIND_SOLVER_MIXED, false, true, many != 0));
    return 0;
}
"""


def test_block_threads(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "probe.cu", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "wind_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    for line in out.strip().splitlines():
        n, solver, many, sie, rk2, tc = (int(v) for v in line.split())
        assert n <= sie <= 256 and sie in (128, 256) and n <= rk2 <= 256 and tc == 256
        if solver == _capi.SOLVERS["gje_f64"] and (n > 64 or not many):
            assert sie == 256


@pytest.mark.gpu
@pytest.mark.parametrize("solver,n", [("gje_f64", 33), ("gje_f64", 64), ("mixed", 65), ("mixed", 112)])
def test_result_does_not_depend_on_the_block(cuda_device, solver, n):
    import torch
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    nsys = sms + 3  # more systems than SMs, and the same ones in two halves
    rng = np.random.default_rng([29, n])
    net = W.random_mass_action(rng, nsys, n, 4 * n, 1e-3, 1e2)
    y0 = rng.uniform(0.0, 1.0, (nsys, n))
    whole = y0.copy()
    _, st, steps = lib.integrate(net, whole, 0.0, 1e-3, 1e-4, 1e-3, "sie", solver, max_attempts=6)
    for part in (slice(0, nsys // 2), slice(nsys // 2, nsys)):
        w = W.Workload(net, y0, 0.0, 1e-3, 1e-4, 1e-3).subset(part)
        y = np.ascontiguousarray(w.y0).copy()
        _, s, c = lib.integrate(w.net, y, 0.0, 1e-3, 1e-4, 1e-3, "sie", solver, max_attempts=6)
        assert np.array_equal(y, whole[part])
        assert np.array_equal(s, st[part]) and np.array_equal(c, steps[part])
