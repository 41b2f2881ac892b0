"""Item costs of a batch (ksim_b200/csrc/batch_plan.h), on the CPU: sliced and
term-record items in one unit, so that kernels are ordered by time."""
from __future__ import annotations

import ctypes
import subprocess

import pytest

from conftest import ROOT

SRC = ROOT / "tests" / "hostemu" / "plan_emu.cpp"
LIB = ROOT / "tests" / "hostemu" / "libksim_plan_emu.so"
CSRC = ROOT / "ksim_b200" / "csrc"


@pytest.fixture(scope="module")
def emu():
    deps = [SRC, *CSRC.glob("*.h")]
    if not LIB.exists() or LIB.stat().st_mtime < max(p.stat().st_mtime for p in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(CSRC), "-o", str(LIB), str(SRC)],
                       check=True)
    L = ctypes.CDLL(str(LIB))
    L.plan_slice_us.restype = L.plan_record_us.restype = ctypes.c_double
    L.plan_slice_us.argtypes = [ctypes.c_int64, ctypes.c_int]
    L.plan_record_us.argtypes = [ctypes.c_double, ctypes.c_int64]
    return L


def test_costs_share_a_unit(emu):
    """A sliced item of many terms outranks a term-record item of few, and the
    other way round; each kind grows with its terms and shots."""
    record = lambda terms, shots: emu.plan_record_us(2000.0 * terms, shots)
    assert emu.plan_slice_us(3000, 1024) > record(20, 256) > emu.plan_slice_us(10, 1024)
    assert record(300, 256) > emu.plan_slice_us(300, 1024)  # the sliced body is the faster one
    w = [emu.plan_slice_us(300, n) for n in (128, 256, 512, 1024)]
    assert w == sorted(w) and record(300, 100) < record(300, 256) < record(301, 256)
