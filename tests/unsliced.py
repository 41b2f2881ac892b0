"""Components that keep the term records.

A sliced stream (ksim_b200/csrc/slice.h) needs every scale 2^(pw + power2) to
be a normal double, so one term scaled below 2^-1022 keeps its whole component
on the term-record kernels, whatever its words and term paths.
"""
from __future__ import annotations

import numpy as np

from ksim_b200 import synth
from ksim_b200.program import FlatComponent


def keep_records(graphs, power2: int = -1100):
    """Scale the first term of the last graph that has one to (almost) nothing."""
    g = [g for g in graphs if len(g.pf_power2)][-1]
    g.pf_power2[0] = power2
    return graphs


# (Tnp, Tph, seed) of graphs whose terms run on 32-bit words; 32-bit and
# hybrid; all term paths
KINDS = {"narrow": (40, 12, 2), "hybrid": (50, 16, 5), "all": (60, 10, 4)}


def component(kind: str, F: int, n_out: int = 3, G: int = 6, sliced: bool = False) -> FlatComponent:
    Tnp, Tph, seed = KINDS[kind]
    rng = np.random.default_rng(seed)
    gs = [synth.random_graph(rng, G, F + k, Tnp, 3, 3, Tph) for k in range(n_out + 1)]
    return FlatComponent(tuple(range(n_out)), np.arange(F, dtype=np.int32), gs if sliced else keep_records(gs))
