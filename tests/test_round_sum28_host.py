"""The panel eigensolver rounds its exact integer level sums to FP64 with round_sum28 and round_wide28
(csrc/exact_round.cuh): built for the host, the nearest double by 128-bit integers."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_round_sum28_is_the_nearest_double(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "round_sum28_check")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "slakonet_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "round_sum28_check.cpp"), "-o", exe])
    out = subprocess.run([exe, "1000000"], capture_output=True, text=True)
    print(out.stdout.strip())
    assert out.returncode == 0 and out.stdout.startswith("0 mismatches")
