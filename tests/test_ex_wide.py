"""The bit-exact collision's integer form (porelb_gb300/csrc/plb_ex.h) at
relaxation times whose forcing factor is small, on both sides of tau = 32
where it gets a scale of its own, at velocities and densities up to the ends
of its domain, and the moments that stand for a node too fast for it: built
for the CPU and checked bit for bit against FP64."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def ex(tmp_path_factory):
    so = tmp_path_factory.mktemp("ex") / "ex_wide_check.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                    "-o", str(so), os.path.join(HERE, "native", "ex_wide_check.cpp")], check=True)
    lib = ctypes.CDLL(str(so))
    lib.ex_wide_check.restype = ctypes.c_long
    lib.ex_wide_check.argtypes = [ctypes.c_long, ctypes.c_ulonglong] + [ctypes.c_double] * 4 + \
        [ctypes.POINTER(ctypes.c_long)] * 2
    lib.mulr_low_check.restype = ctypes.c_long
    lib.mulr_low_check.argtypes = [ctypes.c_long, ctypes.c_ulonglong]
    return lib


def test_small_products(ex):
    assert ex.mulr_low_check(300_000, 5) == 0


def check(ex, n, seed, lo, hi, fmax, umax):
    inside, fast = ctypes.c_long(0), ctypes.c_long(0)
    wrong = ex.ex_wide_check(n, seed, lo, hi, fmax, umax, ctypes.byref(inside),
                             ctypes.byref(fast))
    assert wrong == 0
    return inside.value / n, fast.value / n


@pytest.mark.parametrize("lo,hi,fmax", [(2.4, 2.6, 1e-3), (31.5, 32.5, 1e-3), (32.0, 64.0, 1e-4),
                                        (64.0, 1e3, 1e-5), (1e3, 1e5, 1e-7), (1e5, 1e10, 1e-13)])
def test_large_relaxation_times(ex, lo, hi, fmax):
    inside, _ = check(ex, 40_000, 7, lo, hi, fmax, 0.07)
    assert inside > 0.9


@pytest.mark.parametrize("lo,hi", [(0.52, 2.0), (0.97, 1.03), (40.0, 400.0)])
def test_moments_of_fast_nodes(ex, lo, hi):
    inside, fast = check(ex, 40_000, 11, lo, hi, 1e-6, 0.4)
    assert inside > 0.3 and fast > 0.05
