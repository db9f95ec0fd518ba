"""Every C function libwind exports has one declaration, in a header that the
definition and its callers include: a caller with a prototype of its own would
link against another signature and misread its arguments."""
import glob
import os
import re
import subprocess

from wind_b200 import lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADERS = [os.path.join(ROOT, "include", "wind.h"), os.path.join(ROOT, "wind_b200", "csrc", "float32.h")]


def _code(path):
    with open(path) as fh:
        return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", fh.read(), flags=re.S))


def test_exported_functions_are_declared_in_a_header():
    out = subprocess.run(["nm", "-D", "--defined-only", lib.library_path()], check=True, capture_output=True,
                         text=True).stdout
    exported = sorted({ln.split()[-1] for ln in out.splitlines() if re.search(r" T wind_\w+$", ln)})
    assert "wind_integrate" in exported and "wind_integrate_f32" in exported
    for name in exported:
        where = [h for h in HEADERS if re.search(rf"\b{name}\s*\(", _code(h))]
        assert len(where) == 1, (name, where)


def test_no_source_declares_an_export_by_hand():
    for path in glob.glob(os.path.join(ROOT, "wind_b200", "csrc", "*.cu")):
        by_hand = re.findall(r'extern\s+"C"\s+[\w\s\*]+?\b(wind_\w+)\s*\([^{};]*\)\s*;', _code(path))
        assert not by_hand, (os.path.basename(path), by_hand)
