"""CPU test of the CTA kernel's reaction records (CtaLayout in
wind_b200/csrc/cta_kernel.cuh), compiled host-side with nvcc: where they are
asked for they are aligned, inside their region and beside nothing else, on both
sides of the largest reaction count; a layout without them (RK2) reserves
nothing for them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include "cta_kernel.cuh"
using namespace wind;
int main() {
    const int caps[2] = {232448 - 1024, ((233472 / 2 - 1024 - 288) & ~127)};
    const int ns[] = {33, 48, 64, 65, 96, 128, 129, 157, 200, 256};
    for (int solver = 0; solver < 3; solver++)
        for (int N : ns)
            for (int R : {0, 1, 7, 10 * N, CTA_REC_MAXR, CTA_REC_MAXR + 1, 65535})
                for (int cap : caps) {
                    const CtaLayout L(N, R, false, solver, cap), O(N, R, false, solver, cap, false, false);
                    printf("%d %d %d %d %d %d %d %d %d %zu %zu %zu %zu %d %zu %d %zu %zu\n", solver, N, R, cap,
                           L.data_in_smem ? L.spc + 8 * R : L.rt, L.rec_cap, L.rec, (int)L.rec_in_smem, L.bytes,
                           L.g_doubles, L.g_rec, L.rec_doubles, L.slot_doubles(), O.rec_cap, O.rec_doubles, O.bytes,
                           O.g_doubles, O.slot_doubles());
                }
    printf("max %d\n", CTA_REC_MAXR);
    return 0;
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("ctarecords")
    src = d / "probe.cu"
    src.write_text(PROBE)
    exe = d / "probe"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "wind_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip().splitlines()
    return int(lines[-1].split()[1]), [[int(v) for v in ln.split()] for ln in lines[:-1]]


def test_record_region(rows):
    most, rows = rows
    seen = set()
    for (solver, n, react, cap, before, rec_cap, rec, in_smem, nbytes, g_doubles, g_rec, rec_doubles, slot,
         _, _, off_bytes, off_g, _) in rows:
        # (every part before the records is where a layout without them has it)
        assert g_doubles == off_g
        if solver == 0 or react > most:
            assert rec_cap == 0 and rec_doubles == 0 and slot == g_doubles and nbytes == off_bytes
            continue
        # a warp's list holds at least the padding to four of 32 species
        assert rec_cap >= 8 * react + 4 * ((n + 31) // 32) * 32
        if in_smem:
            assert rec % 16 == 0 and rec >= before and rec == off_bytes
            assert rec + 12 * rec_cap <= nbytes <= cap
            assert rec_doubles == 0 and slot == g_doubles
        else:
            assert nbytes == off_bytes
            # rates of 8 bytes, then species of 4, behind the slot's other parts
            assert g_rec % 2 == 0 and g_rec >= g_doubles
            assert 8 * rec_doubles >= 12 * rec_cap and slot == g_rec + rec_doubles
        seen.add((solver, in_smem))
    assert seen == {(1, 0), (1, 1), (2, 0), (2, 1)}


def test_layout_without_records(rows):
    for row in rows[1]:
        off_cap, off_doubles, off_bytes, off_g, off_slot = row[13:]
        assert off_cap == 0 and off_doubles == 0 and off_slot == off_g
        assert off_bytes <= row[8]
