"""The Fermi search's quotients (skn_quotient, skn_over of csrc/exact_round.cuh), built for the host: rounded as a / b is."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_quotients_are_rounded_once(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "quotient_check")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "slakonet_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "quotient_check.cpp"), "-o", exe])
    out = subprocess.run([exe, "2000000"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
