"""Host calls over sliced kernels at the seams of their SM-filling chunks."""
from __future__ import annotations

import numpy as np
import pytest

from ksim_b200 import synth
from test_gpu_hostio import _device_once

pytestmark = pytest.mark.gpu


def test_filling_chunks_equal_one_launch(cuda_device, oracle_port):
    import torch
    from ksim_b200.sampler import B200ProgramSampler
    u = 512 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(17)
    prog = synth.single_component_program(synth.random_component(rng, n_out=6, F=10, t=8, f_prob=0.05))
    s = B200ProgramSampler(prog, device=0)
    for B in (u, u + u // 4, u + u // 4 + 1, 2 * u + 1, 3 * u + u // 2):
        f = synth.sample_f(rng, B, 10, 0.05)
        for mode in (0, 1):
            got = s.sample(f, B, rng_mode=mode)
            assert np.array_equal(got, _device_once(s, f, B, mode)), (B, mode)
        for lo in range(u - 100, B - 100, u):
            want = oracle_port.program_sample(prog, f[lo:lo + 200], B, rng_mode=1, shot_offset=lo)
            assert np.array_equal(got[lo:lo + 200], want), (B, lo)
