"""The step tail's device code run on the host (tests/cxx/tail_host_test.cpp): a read that no
comparison of results can show ends the program there, and its energy solve meets the update's
at chosen temperatures."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from common import eos9

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


RU = 8.31446261815324e7
U = 2.0 ** -53


def _terms(eos, tmid, T, y):
    """(M, e, Mcv, cv, |dcv/dT|) of the mixture at T: the sums of the terms' magnitudes and of
    the terms of the energy and of its derivative."""
    a = np.where((T < tmid)[:, None], np.asarray(eos.a_lo).reshape(9, 7), np.asarray(eos.a_hi).reshape(9, 7))
    a = a * (RU / np.asarray(eos.mw))[:, None]
    a[:, 0] -= RU / np.asarray(eos.mw)
    i = np.arange(5)
    e = np.concatenate([a[:, 5:6], a[:, :5] * T ** (i + 1) / (i + 1)], axis=1)
    cv = a[:, :5] * T ** i
    dcv = a[:, 1:5] * i[1:] * T ** (i[1:] - 1)
    w = np.asarray(y)[:, None]
    return abs(w * e).sum(), (w * e).sum(), abs(w * cv).sum(), (w * cv).sum(), abs((w * dcv).sum())


@pytest.mark.parametrize("spread", [0.0, 25.0])
def test_the_tails_energy_solve_equals_the_updates(exe, tmp_path, spread):
    """Solutions and first iterates on either side of the range switch and at it. With one
    switch temperature the tail solves on the mixture's polynomial: its coefficients' sums
    (9 terms) and its Horner form (11 operations) leave 21 U of the terms' magnitude, as the
    species' sums do, and the last Newton step is below 1e-10, its square below rounding. With
    several switch temperatures both take the species' sums, bit for bit."""
    eos = eos9()
    t0 = float(np.asarray(eos.tmid)[0])
    tmid = np.asarray(eos.tmid, dtype=float) + spread * np.arange(9)
    rng = np.random.default_rng(12)
    states, want = [], []
    for T in (350.0, t0 - 60.0, t0 - 3.0, t0 + 3.0, t0 + 60.0, 2800.0):
        for guess in (300.0, t0 - 1.0, np.nextafter(t0, 0.0), t0, t0 + 1.0, 2500.0, 0.0, -5.0):
            y = rng.uniform(0.05, 1.0, 9)
            y /= y.sum()
            M, e, Mcv, cv, dcv = _terms(eos, tmid, T, y)
            states.append([e, guess, *y])
            want.append((T, M, Mcv, cv, dcv))
    path = tmp_path / "states"
    with open(path, "wb") as f:
        for a in (eos.mw, tmid, eos.a_lo, eos.a_hi):
            np.ascontiguousarray(a, dtype=np.float64).tofile(f)
        np.array([len(states)], dtype=np.int32).tofile(f)
        np.array(states).tofile(f)
    r = subprocess.run([exe, "energy", str(path)], capture_output=True, text=True, timeout=60, check=True)
    got = np.array([[float(v) for v in ln.split()] for ln in r.stdout.splitlines()])
    assert got.shape == (len(states), 4)
    for (fused, plain, dt_fused, dt_plain), (T, M, Mcv, cv, dcv) in zip(got, want):
        if spread:
            assert fused == plain and dt_fused == dt_plain
            continue
        tol = 2 * 21 * U * M / cv + 4 * U * T
        assert abs(fused - plain) <= tol, (T, fused, plain)
        # e itself is rounded at the states' kinetic energy, 2.6e6 of it
        assert abs(plain - T) <= tol + 8 * U * (M + 2.7e6) / cv, (T, plain)
        # the sound speed's square is T (1 + rmix / cv): half its relative change, with cv from 21 U
        rel = tol / T * (1.0 + T * dcv / cv) + 2 * 21 * U * Mcv / cv + 16 * U
        assert abs(dt_fused - dt_plain) <= rel * dt_plain, (T, dt_fused, dt_plain)
