"""The arena allocator of the batch (host build of the header it uses)."""
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_ranges_stay_apart_and_in_place(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = tmp_path / "range_allocator_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", str(ROOT / "opencafemol_gb300" / "csrc"),
                    str(ROOT / "tests" / "range_allocator_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
