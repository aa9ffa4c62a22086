"""The MPI program's double chains decided in FP32 (geophysics_gb300/csrc/
ziv.cuh), built for the host and compared with the double arithmetic they
stand for: every decided value has the same bits (sign of zero included)
over 6 million chains and squares -- ordinary ranges, cancellation, results
next to a float rounding boundary, subnormal operands and results."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_decided_chains_match_double(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "ziv_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(ROOT, "tests", "ziv_host_check.cpp"),
                    "-o", exe], check=True)
    bad, n, open_, usual, tiny_open, tiny, _ = map(
        int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and n == 12000000
    # the bound leaves about 2^-19 of ordinary values and, of what reaches
    # the second stage, those next to a rounding boundary
    assert open_ <= usual * 2.0 ** -15, (open_, usual)
    assert tiny_open <= 0.2 * tiny, (tiny_open, tiny)
