"""The library's memory pool belongs to a context: contexts that take turns keep
their own, and a device reset, which takes the pool with the old context, leaves
the library usable (in a process of its own)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

TURNS = r"""
import ctypes as C
import numpy as np
from wind_b200 import lib, networks as W
cu = C.CDLL("libcuda.so.1")
def ok(code):
    assert code == 0, code
w = W.workload_katz96(200000)
def run():
    y = w.y0.copy()
    lib.integrate(w.net, y, 0.0, 1e3, 1e-2, 1e-2, "rk2", max_attempts=2)
    return y
want = run()
first, second, dev = C.c_void_p(), C.c_void_p(), C.c_int()
ok(cu.cuCtxGetCurrent(C.byref(first)))
ok(cu.cuDeviceGet(C.byref(dev), 0))
ok(cu.cuCtxCreate_v2(C.byref(second), 0, dev))
free, total = C.c_size_t(), C.c_size_t()
seen = []
for turn in range(12):
    for ctx in (second, first):
        ok(cu.cuCtxSetCurrent(ctx))
        assert np.array_equal(run(), want)
    ok(cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)))
    seen.append(free.value)
# one call takes 24 MB, which a pool of its own per turn would keep each time
grown = seen[1] - seen[-1]
assert grown < 64 << 20, [s >> 20 for s in seen]
ok(cu.cuCtxDestroy_v2(second))
print("turns ok")
"""

RESET = r"""
import ctypes as C
import numpy as np
from wind_b200 import lib, networks as W
w = W.workload_katz96(3000)
rng = np.random.default_rng(3)
mass = W.random_mass_action(rng, 50, 16, 160, 1e-3, 1e1)
ym = rng.uniform(0.0, 1.0, (50, 16))
def run():
    y, z = w.y0.copy(), ym.copy()
    lib.integrate(w.net, y, 0.0, 1e10, 1e-2, 1e-2)
    lib.integrate(mass, z, 0.0, 1e-4, 1e-3, 1e-3, solver="auto")
    return y, z
want = run()
rt = C.CDLL(RUNTIME)
for _ in range(3):
    assert rt.cudaDeviceReset() == 0
    got = run()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
print("reset ok")
"""


def _run(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout


def test_contexts_in_turn_keep_their_pools(cuda_device):
    assert "turns ok" in _run(TURNS)


def test_device_reset(cuda_device):
    from wind_b200 import lib
    # the runtime libwind itself is linked against
    out = subprocess.run(["ldd", lib.library_path()], capture_output=True, text=True).stdout
    names = [ln.split()[0] for ln in out.splitlines() if "libcudart" in ln]
    if not names:
        pytest.skip("libwind has its CUDA runtime inside")
    assert "reset ok" in _run(RESET.replace("RUNTIME", repr(names[0])))
