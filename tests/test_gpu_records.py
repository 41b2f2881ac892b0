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
