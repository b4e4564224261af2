"""CPU: the places in a stored spectral point that the tensor-core contractions
of the packed layout read (egx_diglayout.cuh), compiled for the host by the system C++ compiler:
every entry of the block matrix is the packed block's of its row and column,
and padded ones stay inside the block, for every layer count it takes."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "extreme_gb300", "csrc")


def test_places_of_the_sub_blocks(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "diglayout_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, "-o", exe, os.path.join(HERE, "diglayout_check.cpp")],
                   check=True)
    lines = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip().splitlines()
    assert lines == ["nz %d errors 0" % nz for nz in range(1, 49)]
