"""The GPU programs' opening-angle bin without its double quotient
(geophysics_gb300/csrc/adcig.cuh), built for the host and compared with the
quotient: the same bin for 4 million pairs, a quarter of them with a tiny,
subnormal or zero denominator."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bins_match_double_quotient(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "adcig_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(ROOT, "tests", "adcig_host_check.cpp"),
                    "-o", exe], check=True)
    bad, n, _ = map(int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and n == 4000000
