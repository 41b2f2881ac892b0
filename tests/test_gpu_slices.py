"""The sliced sampling kernel (csrc/slice_tile.cuh) at the edges of its tile
shapes, parameter counts and term kinds, bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import same_bits
from ksim_b200 import synth
from ksim_b200.program import FlatComponent, FlatProgram
from test_gpu_parity import _component, device_sample

pytestmark = pytest.mark.gpu


def _graphs(seed, F, n_out, G=3, **kw):
    rng = np.random.default_rng(seed)
    size = dict(Tnp=9, Thp=4, Tpp=3, Tph=3, **kw)
    return rng, [synth.random_graph(rng, G, F + k, **size) for k in range(n_out + 1)]


@pytest.mark.parametrize("F", [5, 16, 140])
def test_tile_shapes(cuda_device, oracle_port, F):
    """Shot counts around each line of the launch rule (140 parameters: one that
    keeps the narrower tile), and every tile width a caller can ask for."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng, graphs = _graphs(F, F, 3)
    top = 2 * sms * 1024 + 65
    f = rng.integers(0, 2, size=(top, F)).astype(np.uint8)
    want, want_amp = oracle_port.PortOracle(graphs, F).sample(f, 9, 0, return_amp=True)
    kc = _component(graphs, F)
    for edge in (1, 64, 128, 1024, sms * 128, sms * 256, sms * 512, sms * 1024, 2 * sms * 1024):
        for B in (edge - 1, edge, edge + 1, edge + 64):
            if B:
                bits, amp = device_sample(kc, f[:B], 9, 0)
                assert np.array_equal(bits, want[:B]) and same_bits(amp, want_amp[:B]), B
    for threads in (32, 64, 128, 256):
        kc.set_launch(threads=threads)
        for B in (4 * threads - 1, 4 * threads + 1, 9001):
            assert np.array_equal(device_sample(kc, f[:B], 9, 0)[0], want[:B]), (threads, B)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("F,n_out", [(0, 1), (1, 7), (3, 4), (4, 9), (17, 8), (33, 16), (246, 8)])
def test_columns(cuda_device, oracle_module, F, n_out, mode):
    """Parameter and output counts around the 4- and 8-column loads and stores
    up to 254 rows; two components with columns out of order and in order."""
    rng, a = _graphs(100 + F, F, n_out)
    b = [synth.random_graph(rng, 2, F + k, 5, 2, 2, 2) for k in range(n_out + 1)]
    for order, sel in ((rng.permutation(2 * n_out), rng.permutation(F + 2)[:F]), (np.arange(2 * n_out), np.arange(F))):
        prog = FlatProgram([FlatComponent(tuple(order[:n_out]), sel.astype(np.int32), a),
                            FlatComponent(tuple(order[n_out:]), np.arange(F, dtype=np.int32), b)],
                           order.astype(np.int64), 2 * n_out, 0)
        from ksim_b200.sampler import B200ProgramSampler
        s = B200ProgramSampler(prog)
        for cols in (F + 2, F + 16 - F % 16 + 16):
            for B in (1, 131, 1500):
                f = rng.integers(0, 2, size=(B, cols)).astype(np.uint8)
                assert np.array_equal(s.sample(f, 21, rng_mode=mode),
                                      oracle_module.program_sample(prog, f, 21, mode)), (cols, B)


@pytest.mark.parametrize("G", [1, 8, 9, 16, 17])
def test_term_kinds(cuda_device, oracle_port, G):
    """Terms with 0 to 15 both-odd columns (narrow, listed classes, tables in
    global memory), dense masks (more than four slots), 1 to 3 chunks."""
    rng = np.random.default_rng(G)
    graphs = [synth.random_graph(rng, G, 10 + k, 45, 2, 2, 15, density=0.4) for k in range(3)]
    for g in graphs[1:]:
        g.ph_alpha[:] = 2 * rng.integers(0, 4, size=g.ph_alpha.shape) + 1
        g.ph_beta[:] = 2 * rng.integers(0, 4, size=g.ph_beta.shape) + 1
        g.ph_counts[:] = np.arange(G) % 16
    kc, po = _component(graphs, 10), oracle_port.PortOracle(graphs, 10)
    f = rng.integers(0, 2, size=(700, 10)).astype(np.uint8)
    for mode in (0, 1):
        want, want_amp = po.sample(f, 4, mode, return_amp=True)
        bits, amp = device_sample(kc, f, 4, mode)
        assert np.array_equal(bits, want) and same_bits(amp, want_amp)
    for k in range(3):
        pv = rng.integers(0, 2, size=(333, 10 + k)).astype(np.uint8)
        assert same_bits(kc.eval(k, pv), po.eval(k, pv))
        assert same_bits(kc.eval_abs(k, pv), po.eval_abs(k, pv))


def test_non_finite_approximation_factor(cuda_device, oracle_port):
    """An infinite factor makes a dead term NaN: amplitudes, bits and the
    status word say so."""
    from ksim_b200 import _abi
    rng, graphs = _graphs(31, 12, 3)
    for g in graphs:
        g.np_phases[:, 0] = 0
        g.pf_has_approx, g.pf_approx = True, np.full(3, 0.5 + 1j, np.complex64)
    graphs[2].pf_approx[1] = np.inf
    kc, po = _component(graphs, 12), oracle_port.PortOracle(graphs, 12)
    f = rng.integers(0, 2, size=(3000, 12)).astype(np.uint8)
    want, want_amp = po.sample(f, 8, 0, return_amp=True)
    bits, amp = device_sample(kc, f, 8, 0)
    assert np.isnan(want_amp).any() and np.array_equal(np.isnan(amp), np.isnan(want_amp))
    assert np.array_equal(bits, want) and kc.status(reset=True) & _abi.FLAG_NAN
    # (the oracle's pairs as they are: its complex array turns infinities into NaN)
    pv = rng.integers(0, 2, size=(333, 14)).astype(np.uint8)
    a = np.zeros((333, 2))
    assert po.L.oracle_eval(po.descs, 4, 2, _abi.u8ptr(pv), 333, 14, a.ctypes.data_as(oracle_port._dp)) == 0
    got = kc.eval_abs(2, pv)
    nan = np.isnan(a).any(1)
    assert np.array_equal(np.isnan(got), nan) and np.array_equal(np.isinf(got), np.isinf(a).any(1) & ~nan)


@pytest.mark.parametrize("G", [4, 5])
def test_tile_shapes_by_terms(cuda_device, oracle_port, G):
    """The shot counts around the launch rule's lines for components with chunks
    of at most four terms, and of more (CTAs of 256 and of 512 threads)."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng, graphs = _graphs(40 + G, 16, 3, G=G)
    f = rng.integers(0, 2, size=(sms * 1024 + 1, 16)).astype(np.uint8)
    want, want_amp = oracle_port.PortOracle(graphs, 16).sample(f, 9, 0, return_amp=True)
    kc = _component(graphs, 16)
    for edge in (1, 128, sms * 128, sms * 256, sms * 512, sms * 1024):
        for B in (edge, edge + 1):
            bits, amp = device_sample(kc, f[:B], 9, 0)
            assert np.array_equal(bits, want[:B]) and same_bits(amp, want_amp[:B]), B
    pv = rng.integers(0, 2, size=(sms * 1024, 18)).astype(np.uint8)
    for B in (100, sms * 256, sms * 512, sms * 1024):
        assert same_bits(kc.eval_abs(2, pv[:B]), oracle_port.PortOracle(graphs, 16).eval_abs(2, pv[:B])), B
