"""The sliced term stream (csrc/slice.cpp) against the oracle, on the CPU.

A test-only walker (tests/hostemu/slice_emu.cpp) evaluates the stream the way
the sampling kernel does; every amplitude double must equal the oracle's
(zx_eval.hpp:101-178 semantics) bit for bit, up to the sign of a zero.
"""
from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from ksim_b200 import synth

CSRC = ROOT / "ksim_b200" / "csrc"
LIB = ROOT / "tests" / "hostemu" / "libksim_slice_emu.so"


@pytest.fixture(scope="module")
def emu():
    from ksim_b200._abi import GraphDesc
    srcs = [ROOT / "tests" / "hostemu" / "slice_emu.cpp", CSRC / "slice.cpp", CSRC / "image.cpp"]
    deps = srcs + list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh"))
    if not LIB.exists() or LIB.stat().st_mtime < max(p.stat().st_mtime for p in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", str(CSRC),
                        "-o", str(LIB), *map(str, srcs)], check=True)
    L = ctypes.CDLL(str(LIB))
    L.slice_emu_info.argtypes = [ctypes.POINTER(GraphDesc), ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    L.slice_emu_eval.argtypes = [ctypes.POINTER(GraphDesc), ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                 ctypes.POINTER(ctypes.c_uint8), ctypes.c_int64, ctypes.c_int64, ctypes.c_void_p]
    L.slice_emu_error.restype = ctypes.c_char_p
    return L


def _descs(graphs):
    from ksim_b200 import _abi
    from ksim_b200.program import graph_to_dict
    return _abi.graphs_to_descs([graph_to_dict(g) for g in graphs])


def info(emu, graphs, F):
    descs, keep = _descs(graphs)
    v = (ctypes.c_int64 * 8)()
    assert emu.slice_emu_info(descs, len(graphs), F, v) == 0, emu.slice_emu_error()
    return dict(zip(("ok", "rows", "planes", "chunks", "bytes", "terms", "wide", "big"), v))


def check(emu, oracle_port, graphs, F, rng, rows=97):
    from ksim_b200 import _abi
    descs, keep = _descs(graphs)
    po = oracle_port.PortOracle(graphs, F)
    for gi, g in enumerate(graphs):
        P = g.np_params.shape[2]
        pv = np.ascontiguousarray(rng.integers(0, 2, size=(rows, P)).astype(np.uint8))
        got = np.zeros((rows, 2))
        assert emu.slice_emu_eval(descs, len(graphs), F, gi, _abi.u8ptr(pv), rows, P, got.ctypes.data) == 0
        want = po.eval(gi, pv)
        assert np.array_equal(got[:, 0] + 0.0, want.real + 0.0) and np.array_equal(got[:, 1] + 0.0, want.imag + 0.0), gi


@pytest.mark.parametrize("seed", range(6))
def test_random_components(emu, oracle_port, seed):
    rng = np.random.default_rng(500 + seed)
    F = int(rng.integers(0, 120))
    comp = synth.random_component(rng, n_out=int(rng.integers(1, 14)), F=F, t=int(rng.integers(1, 20)), f_prob=0.05)
    assert info(emu, comp.graphs, F)["ok"]
    check(emu, oracle_port, comp.graphs, F, rng)


@pytest.mark.parametrize("Tnp,Thp,Tpp,Tph", [(0, 0, 0, 0), (1, 1, 1, 1), (4, 5, 2, 3), (40, 9, 7, 31), (70, 0, 0, 14),
                                             (90, 4, 4, 2)])
def test_every_column_kind(emu, oracle_port, Tnp, Thp, Tpp, Tph):
    """All phases and coefficients (odd HalfPi coefficients too), dense and
    empty masks, approximation factors, counts of zero and below; up to 15
    columns of the primes above 3, tables beyond the staged size."""
    rng = np.random.default_rng(Tnp + 100 * Tph)
    gs = [synth.random_graph(rng, 5, 12 + k, Tnp, Thp, Tpp, Tph, density=0.3) for k in range(3)]
    for g in gs:
        g.np_phases[:] = rng.integers(0, 8, size=g.np_phases.shape) if Tnp < 60 else g.np_phases
        g.hp_coeffs[:] = rng.integers(0, 8, size=g.hp_coeffs.shape)
        g.np_params[:, ::5] = 0
        g.pf_approx = (rng.normal(size=5) + 1j * rng.normal(size=5)).astype(np.complex64)
        g.pf_has_approx = True
        g.np_counts[0] = -2
    n = info(emu, gs, 12)
    if n["ok"]:
        check(emu, oracle_port, gs, 12, rng)
    assert n["ok"] or Tph == 31


def test_phase_pair_classes(emu, oracle_port):
    """One term per (alpha, beta) pair, and terms of 4 to 15 both-odd columns
    (classes listed by a table; value tables beyond the staged size)."""
    rng = np.random.default_rng(64)
    g = synth.random_graph(rng, 64, 10, 6, 2, 2, 1, density=0.3)
    g.ph_alpha[:, 0], g.ph_beta[:, 0], g.ph_counts[:] = np.arange(64) // 8, np.arange(64) % 8, 1
    h = synth.random_graph(rng, 12, 11, 50, 2, 2, 15, density=0.3)
    h.ph_alpha[:] = 2 * rng.integers(0, 4, size=h.ph_alpha.shape) + 1
    h.ph_beta[:] = 2 * rng.integers(0, 4, size=h.ph_beta.shape) + 1
    h.ph_counts[:] = np.arange(4, 16)
    n = info(emu, [g, h], 10)
    assert n["ok"] and n["wide"] == 11 and n["big"] > 0
    check(emu, oracle_port, [g, h], 10, rng, rows=400)


def test_not_sliced(emu):
    """Terms without a proof (int64 may wrap; scales beyond the normal range),
    more than 126 lambda rows, more than 254 parameters."""
    rng = np.random.default_rng(3)
    wrap = synth.random_graph(rng, 1, 10, 250, 0, 0, 0)
    wrap.np_phases[:], wrap.np_counts[:] = 1, 250
    assert not info(emu, [wrap], 10)["ok"]
    scale = synth.random_graph(rng, 1, 10, 4, 1, 1, 1)
    scale.pf_power2[:] = 1023
    assert not info(emu, [scale], 10)["ok"]
    assert info(emu, [synth.random_graph(rng, 1, 254, 4, 1, 1, 1)], 254)["ok"]
    assert not info(emu, [synth.random_graph(rng, 1, 255, 4, 1, 1, 1)], 255)["ok"]
    empty = synth.random_graph(rng, 0, 10, 4, 1, 1, 1)
    assert info(emu, [empty], 10) == {"ok": 1, "rows": 10, "planes": 0, "chunks": 1, "bytes": 48, "terms": 0,
                                      "wide": 0, "big": 0}


@pytest.mark.parametrize("factor", [complex(np.inf, 0.0), complex(0.0, -np.inf), complex(np.nan, 1.0)])
def test_non_finite_approximation_factor(emu, factor):
    """A dead term (value 0) times a factor that is not finite is NaN
    (zx_eval.hpp:177-178), which the zero row of a value table is not: the
    component keeps the term records."""
    rng = np.random.default_rng(9)
    g = synth.random_graph(rng, 3, 10, 4, 2, 2, 2)
    g.np_phases[:, 0] = 0  # a row that kills the term
    g.pf_has_approx = True
    g.pf_approx = np.full(3, 1.5 - 0.25j, np.complex64)
    assert info(emu, [g], 10)["ok"]
    g.pf_approx[1] = factor
    assert not info(emu, [g], 10)["ok"]
    g.pf_has_approx = False  # the factors are not read
    assert info(emu, [g], 10)["ok"]


@pytest.mark.parametrize("n", [24, 60, 86, 112])
def test_many_products_of_two_plus_two_i(emu, oracle_port, n):
    """PhasePairs columns with both phases 2 and equal signs contribute
    (2 + 2i)^n: 2^(1.5 n) before its powers of two are taken out, past 127
    bits from n = 85."""
    rng = np.random.default_rng(n)
    g = synth.random_graph(rng, 2, 10, 4, 1, 1, n, density=0.3)
    g.ph_alpha[:], g.ph_beta[:], g.ph_counts[:], g.np_phases[:] = 2, 2, n, 1
    g.ph_alpha_p[:], g.ph_beta_p[:] = 0, 0
    assert info(emu, [g], 10)["ok"]
    check(emu, oracle_port, [g], 10, rng)


def test_stream_size_bound(emu):
    """A stream beyond the bound is not built (its component keeps the term
    records); tables kept in global memory count too."""
    rng = np.random.default_rng(11)
    gs = [synth.random_graph(rng, 6, 10 + k, 45, 2, 2, 15, density=0.4) for k in range(3)]
    for g in gs:
        g.ph_alpha[:] = 2 * rng.integers(0, 4, size=g.ph_alpha.shape) + 1
        g.ph_beta[:] = 2 * rng.integers(0, 4, size=g.ph_beta.shape) + 1
        g.ph_counts[:] = 15
    descs, keep = _descs(gs)
    f = emu.slice_emu_bytes
    f.restype, f.argtypes = ctypes.c_int64, [*emu.slice_emu_info.argtypes[:3], ctypes.c_int64]
    full = f(descs, 3, 10, 1 << 30)
    assert info(emu, gs, 10)["big"] == 18 and full == info(emu, gs, 10)["bytes"] > 18 * 16384
    assert f(descs, 3, 10, full) == full and f(descs, 3, 10, full - 16384) == 0 and f(descs, 3, 10, 0) == 0


@pytest.mark.parametrize("kind", ["narrow", "hybrid", "all"])
@pytest.mark.parametrize("F", [20, 100, 160, 240])
def test_components_kept_on_term_records(emu, kind, F):
    """The components the GPU tests of the term-record kernels use have no sliced
    stream, and the term paths they are named for; the same graphs without the
    scaled-down term have one."""
    import unsliced
    from ksim_b200.perfmodel import component_work
    comp = unsliced.component(kind, F)
    w = component_work(comp)
    paths = [w["hybrid_terms"] > 0, w["wide_terms"] + w["exact_terms"] > 0]
    assert paths == {"narrow": [False, False], "hybrid": [True, False], "all": [True, True]}[kind]
    assert not info(emu, comp.graphs, F)["ok"]
    assert info(emu, unsliced.component(kind, F, sliced=True).graphs, F)["ok"]
