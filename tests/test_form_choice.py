"""The choice between two forms of a solve: the estimate of a mode's step attempts and what a launch's modes
make of it (form_choice.cuh compiled for the host)."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def choice(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("shim") / "form_choice_shim.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-I", os.path.join(ROOT, "disco-eb_b200", "csrc"),
                    "-o", out, os.path.join(ROOT, "tests", "cpu_model", "form_choice_shim.cpp")], check=True)
    S = ctypes.CDLL(out)
    S.shim_attempts.argtypes = [ctypes.c_double, ctypes.c_int]
    S.shim_attempts.restype = ctypes.c_longlong
    S.shim_short_chain_wins.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
    S.shim_choice.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.POINTER(ctypes.c_int)]
    return S


def _wins(S, k, limit, n_out=1):
    k = np.ascontiguousarray(k, dtype=np.float64)
    return bool(S.shim_short_chain_wins(len(k), k.ctypes.data, n_out, limit))


def test_attempts_follow_the_measured_counts(choice):
    # step attempts of P(k) solves at rtol 1e-5
    for k, n in ((1e-4, 77), (1e-3, 145), (1e-2, 360), (0.1, 345), (0.5, 362), (1.0, 450), (3.0, 860), (10.0, 1410)):
        assert abs(choice.shim_attempts(k, 0) / 10 / n - 1) < 0.1, k
    assert choice.shim_attempts(0.1, 320) - choice.shim_attempts(0.1, 0) == 3 * 320
    k = np.geomspace(1e-5, 100.0, 4000)  # no jump within or between octaves
    a = np.array([choice.shim_attempts(float(x), 0) for x in k])
    assert (a > 0).all() and (np.abs(np.diff(a)) <= 0.02 * a[:-1]).all()


@pytest.mark.parametrize("k", [0.0, -1.0, 5e-324, math.inf, math.nan])
def test_attempts_of_any_number_stay_in_the_table(choice, k):
    assert 700 <= choice.shim_attempts(k, 0) <= 35700


def test_modes_of_equal_length_count_as_they_are(choice):
    k = np.full(100, 0.37)
    assert _wins(choice, k, 100) and not _wins(choice, k, 99)


def test_spread_modes_count_less_in_any_order(choice):
    k = np.geomspace(1e-4, 5.0, 1000)
    need = min(n for n in range(1, 1001) if _wins(choice, k, n))
    assert 300 < need < 340
    for order in (k[::-1], np.random.default_rng(0).permutation(k)):
        assert _wins(choice, order, need) and not _wins(choice, order, need - 1)
    assert not _wins(choice, k, need, n_out=2000)  # outputs make modes alike


def test_launch_asks_the_wavenumbers_between_one_and_four_limits(choice):
    gate = ctypes.c_int()
    for n, forms, g in ((100, 1, -1), (101, 3, 100), (400, 3, 100), (401, 2, -1)):
        assert choice.shim_choice(n, 100, ctypes.byref(gate)) == forms and gate.value == g
    assert choice.shim_choice(2**31 - 1, 2**31 - 1, ctypes.byref(gate)) == 1
