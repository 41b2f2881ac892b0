"""The term-record kernels (components without a sliced stream) beside the
sliced ones, bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import unsliced
from helpers import same_bits
from ksim_b200 import synth
from test_gpu_parity import _component, device_sample

pytestmark = pytest.mark.gpu


WORDS = (20, 100, 160, 240)  # f parameters of components of W = 1, 2, 3, 4


@pytest.mark.parametrize("kind", unsliced.KINDS)
@pytest.mark.parametrize("F", WORDS)
def test_sampling_kernels(cuda_device, oracle_port, kind, F):
    """k_sample of every width and set of term paths, staged or not, at the
    smallest and a large slot, both streams, with an offset."""
    comp = unsliced.component(kind, F)
    kc, po = _component(comp.graphs, F), oracle_port.PortOracle(comp.graphs, F)
    assert kc.words == 1 + WORDS.index(F)
    rng = np.random.default_rng(F)
    f = rng.integers(0, 2, size=(1300, F)).astype(np.uint8)
    for mode, off in ((0, 0), (1, 777)):
        want, want_amp = po.sample(f, 123, mode, return_amp=True, shot_offset=off)
        bits, amp = device_sample(kc, f, 123, mode, shot_offset=off)
        assert np.array_equal(bits, want) and same_bits(amp, want_amp), (mode, off)
    want = po.sample(f, 9, 0)
    smallest = (kc.stats()["max_term_bytes"] + 15) // 16 * 16
    for threads in (32, 128, 256):
        for staged, slot in ((0, 16384), (1, smallest), (1, 32768)):
            kc.set_launch(threads=threads, staged=staged, slot_bytes=slot)
            assert np.array_equal(device_sample(kc, f, 9, 0)[0], want), (threads, staged, slot)
    pv = rng.integers(0, 2, size=(65, F + 2)).astype(np.uint8)
    assert same_bits(kc.eval(2, pv), po.eval(2, pv)) and same_bits(kc.eval_abs(2, pv), po.eval_abs(2, pv))


def test_wait_timeouts(cuda_device, oracle_port):
    """A staging wait of a term-record kernel that runs out: the host call
    reports it, a batch raises the flag and leaves the shots; both are exact
    afterwards."""
    from ksim_b200._abi import FLAG_WAIT_TIMEOUT
    comp = unsliced.component("narrow", 100, n_out=12)
    kc, po = _component(comp.graphs, 100), oracle_port.PortOracle(comp.graphs, 100)
    f = synth.sample_f(np.random.default_rng(4), 5000, 100, 0.1)
    kc.set_wait_limit(1)
    with pytest.raises(TimeoutError, match="staging wait"):
        kc.sample(f, 5)
    kc.set_wait_limit(0)
    assert not kc.status() & FLAG_WAIT_TIMEOUT and np.array_equal(kc.sample(f, 5), po.sample(f, 5, 0))

    progs, fs, bs = _batch([comp], [5000])
    bc = bs.samplers[0].components[0][1]
    bc.set_wait_limit(1)
    bs._build(bs.tuning)  # (a batch takes the bound in force when it is created)
    bs.d_out[0].fill_(9)
    bs.set_inputs(fs)
    bs.launch()
    assert (bs.results()[0] == 9).any() and bc.status(reset=True) & FLAG_WAIT_TIMEOUT
    bc.set_wait_limit(0)
    bs._build(bs.tuning)
    assert np.array_equal(bs.sample(fs)[0], oracle_port.program_sample(progs[0], fs[0], 0))
    assert not bc.status() & FLAG_WAIT_TIMEOUT  # (these inputs do reach prev <= 0)


def _batch(comps, shots, seed=1):
    from ksim_b200.batch import BatchSampler
    progs = [synth.single_component_program(c) for c in comps]
    F = [len(c.f_selection) for c in comps]
    rng = np.random.default_rng(seed)
    fs = [synth.sample_f(rng, b, n, 0.1) for b, n in zip(shots, F)]
    return progs, fs, BatchSampler(progs, shots, seeds=list(range(len(progs))), n_f=F)


def test_batch_class_with_and_without_sliced_streams(cuda_device, oracle_port):
    """Two jobs of one (W, term paths) class, one of them without a sliced
    stream: each takes its own body (two launches, tiles of 256 shots and of
    up to 1,024), and either alone is one launch."""
    shots = [5000, 3001]
    comps = [unsliced.component("narrow", 60, sliced=True), unsliced.component("narrow", 60)]
    progs, fs, bs = _batch(comps, shots)
    assert bs.info()["launches"] == 2
    for i, got in enumerate(bs.sample(fs)):
        assert np.array_equal(got, oracle_port.program_sample(progs[i], fs[i], i)), i
    records = -(-shots[1] // 256)
    assert records + -(-shots[0] // 1024) <= bs.info()["items"] <= records + -(-shots[0] // 256)
    for i in (0, 1):
        assert _batch(comps[i:i + 1], shots[i:i + 1])[2].info()["launches"] == 1


@pytest.mark.parametrize("per_sm", [0, 1])
def test_batch_ctas_per_sm(cuda_device, oracle_port, per_sm):
    """ctas_per_sm bounds the persistent CTAs of the sliced jobs together,
    whichever of their classes they belong to."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    comps = [unsliced.component(k, F, sliced=True) for k, F in (("narrow", 20), ("hybrid", 60), ("all", 60), ("all", 124))]
    progs, fs, bs = _batch(comps, [200_000] * 4)
    bs._build({"threads": 128, "slot_bytes": 14336, "ctas_per_sm": per_sm})
    assert bs.info()["launches"] == 4
    assert bs.info()["grid"] == (2 - per_sm) * sms
    for i, got in enumerate(bs.sample(fs)):
        assert np.array_equal(got[:3000], oracle_port.program_sample(progs[i], fs[i][:3000], i)), i
        rest = bs.samplers[i].sample(fs[i], i)
        assert np.array_equal(got, rest), i


def test_served_term_records_stay_in_the_loop(cuda_device, oracle_port):
    """Programs of up to 256 parameter bits without a sliced stream run in the
    device loop beside sliced ones (every W and set of term paths), bit for
    bit; none is a plain launch, which would wait for the loop to go idle."""
    from ksim_b200.serve import Server
    rng = np.random.default_rng(5)
    reqs = []
    for k in unsliced.KINDS:
        for F in (20, 60, 124, 188, 250):  # W = 1, 2 (61 + 3 parameters), 2, 3, 4
            for sliced in (False, True):
                prog = synth.single_component_program(unsliced.component(k, F, sliced=sliced))
                for B in (1, 513, 2000):
                    reqs.append((prog, synth.sample_f(rng, B, F, 0.1), len(reqs)))
    with Server(device=0, idle_us=2000) as srv:
        handles = [srv.submit(p, f, seed) for p, f, seed in reqs]
        got = [h.result(timeout=120) for h in handles]
        st = srv.stats()
    assert st["failed"] == 0 and st["completed"] == len(reqs) and st["side_launches"] == 0
    for (p, f, seed), g in zip(reqs, got):
        assert np.array_equal(g, oracle_port.program_sample(p, f, seed))


def test_batch_kernels(cuda_device, oracle_port):
    """A batch of term-record jobs of every width and set of term paths beside
    sliced jobs of the same classes: a kernel each, every result exact."""
    comps, shots = [], []
    for kind in unsliced.KINDS:
        for i, F in enumerate(WORDS):
            for sliced in (False, True):
                comps.append(unsliced.component(kind, F, sliced=sliced))
                shots.append(700 + 301 * i)
    progs, fs, bs = _batch(comps, shots)
    assert bs.info()["launches"] == 2 * len(unsliced.KINDS) * len(WORDS)
    want = [oracle_port.program_sample(p, f, i) for i, (p, f) in enumerate(zip(progs, fs))]
    for tuning in ({"threads": 128, "slot_bytes": 14336, "ctas_per_sm": 0},
                   {"threads": 64, "slot_bytes": 8192, "ctas_per_sm": 1},
                   {"threads": 256, "slot_bytes": 16384, "ctas_per_sm": 2}):
        bs._build(tuning)
        for i, got in enumerate(bs.sample(fs)):
            assert np.array_equal(got, want[i]), (tuning, i)
