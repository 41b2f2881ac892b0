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
