"""Tables of the 60-bit fixed-point kernel, checked on the host
(tests/cxx/fx_tables_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "solidfmm_gb300", "csrc")


def test_fx_tables(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "fx_tables"
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cxx", "fx_tables_check.cpp"), os.path.join(CSRC, "sfmm_tables.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout
