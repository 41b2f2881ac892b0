"""Host plans, on the CPU: the item costs of a batch (ksim_b200/csrc/batch_plan.h:
sliced and term-record items in one unit, so that kernels are ordered by time)
and the chunks of a host call over sliced kernels (hostio.h), and the widths of sliced
tiles (slice.h)."""
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


SMS = 148
U = 512 * SMS  # shots that fill the SMs once


def _bounds(emu, B, in_row, out_row, terms, graphs, sliced=1):
    out = (ctypes.c_int64 * 4096)()
    i64 = ctypes.c_int64
    n = emu.plan_host_call(i64(B), i64(in_row), i64(out_row), sliced, i64(terms), i64(graphs), i64(SMS), out, 4096)
    return list(out[:n])


def _ramp(emu, B, row):
    out = (ctypes.c_int64 * 4096)()
    return list(out[:emu.plan_host_ramp(ctypes.c_int64(B), ctypes.c_int64(row), out, 4096)])


@pytest.mark.parametrize("B", [1, U - 1, U, U + 1, U + U // 4, U + U // 4 + 1, 2 * U, 2 * U + U // 4 + 1, 400_000])
def test_filling_chunks(emu, B):
    """Kernels that outlast the copies: chunks of U, the last up to a quarter
    more, never less than a quarter."""
    b = _bounds(emu, B, 8, 2, 2000, 50)
    assert b[0] == 0 and b[-1] == B and all(x < y for x, y in zip(b, b[1:]))
    assert all(y - x == U for x, y in zip(b[:-2], b[1:-1]))
    assert b[-1] - b[-2] <= U + U // 4 and (len(b) == 2 or b[-1] - b[-2] > U // 4)


def test_which_plan(emu):
    """Copies of more than four kernel latencies, few-term calls of one chunk
    with many output bytes, and components without a sliced stream take the
    ramp; the other calls take filling chunks."""
    for B, in_row, out_row, terms, graphs, ramp in (
            (1_000_000, 64, 40, 306, 41, True), (400_000, 64, 40, 306, 41, False), (300_000, 0, 40, 306, 41, False),
            (75_000, 60, 60, 61, 61, True), (75_000, 64, 20, 21, 21, False), (75_000, 20, 200, 201, 201, False),
            (50_000, 200, 5, 6, 6, False), (20_011, 64, 40, 306, 41, False),
            (20_000, 20, 200, 201, 201, False), (100_000, 0, 5, 20, 6, False)):
        got, want = _bounds(emu, B, in_row, out_row, terms, graphs), _ramp(emu, B, in_row + out_row)
        assert (got == want) == ramp or len(want) == 2, (B, in_row, out_row, terms)
        assert _bounds(emu, B, in_row, out_row, terms, graphs, sliced=0) == want


def test_tile_widths(emu):
    """The widths the launches choose pass; those a warp of lanes would not fill,
    or a CTA would not cover, are refused on the host."""
    ok = [(1, 128, 512), (1, 256, 512), (1, 512, 512), (4, 1024, 512), (4, 1024, 256), (8, 2048, 256),
          *((4, 4 * t, t) for t in (32, 64, 128, 256)), *((4, n, 256) for n in (128, 256, 512))]
    bad = [(4, 64, 256), (4, 32, 256), (4, 96, 256), (4, 192, 256), (4, 2048, 512), (4, 512, 64), (8, 1024, 256),
           (8, 4096, 512), (1, 32, 512), (1, 1024, 512), (1, 0, 512)]
    assert [x for x in ok if not emu.plan_tile_ok(*x)] == [] and [x for x in bad if emu.plan_tile_ok(*x)] == []


def test_tuner_shapes():
    """Without term-record jobs the autotuner times each distinct shape once."""
    from ksim_b200.batch import _CANDIDATES, _shapes
    assert _shapes(False) == _CANDIDATES
    got = [(c["threads"] <= 64, c["slot_bytes"]) for c in _shapes(True)]
    assert sorted(got) == [(False, 16384), (True, 16384)]
