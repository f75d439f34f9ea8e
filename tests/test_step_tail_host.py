"""The step tail's device code run on the host (tests/cxx/tail_host_test.cpp), where a read
that no comparison of results can show ends the program."""
import os
import shutil
import subprocess

import pytest

CXX = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cxx")
EXE = os.path.join(CXX, "_build", "tail_host_test")


@pytest.fixture(scope="module")
def exe():
    if shutil.which("g++") is None or not os.path.exists("/usr/local/cuda/include/cuda_runtime.h"):
        pytest.skip("g++ or the CUDA headers are missing")
    subprocess.run(["make", "-s", "-C", CXX, EXE], check=True)
    return EXE


def test_the_tail_reads_no_other_cells_state(exe):
    """The tail replaces the state in place, its blocks in no order: every other cell's tail
    runs with the region's first row of cells unreadable, on FP32 and on FP64 fluxes."""
    r = subprocess.run([exe, "cells"], timeout=60)
    assert r.returncode == 0, f"exit status {r.returncode} (-11: the tail read another cell's state)"
