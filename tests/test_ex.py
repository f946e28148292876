"""The bit-exact collision's integer form (porelb_gb300/csrc/plb_ex.h), built
for the CPU and checked bit for bit against the same operations in FP64: over
every kind of relaxation time it treats apart, velocities and densities past
the ends of its domain, values with short significands and at the weights.
What it reports as outside has to leave most near-equilibrium nodes in."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def ex(tmp_path_factory):
    so = tmp_path_factory.mktemp("ex") / "ex_check.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                    "-o", str(so), os.path.join(HERE, "native", "ex_check.cpp")], check=True)
    lib = ctypes.CDLL(str(so))
    lib.ex_check.restype = ctypes.c_long
    lib.ex_check.argtypes = [ctypes.c_long, ctypes.c_ulonglong, ctypes.c_int,
                             ctypes.POINTER(ctypes.c_long)]
    lib.mulr_check.restype = ctypes.c_long
    lib.mulr_check.argtypes = [ctypes.c_long, ctypes.c_ulonglong]
    return lib


@pytest.mark.parametrize("tau_mode", range(6))
def test_collision_equals_fp64(ex, tau_mode):
    inside = ctypes.c_long(0)
    assert ex.ex_check(100_000, 1000 + tau_mode, tau_mode, ctypes.byref(inside)) == 0
    assert inside.value > 60_000


def test_rounded_product(ex):
    assert ex.mulr_check(300_000, 5) == 0
