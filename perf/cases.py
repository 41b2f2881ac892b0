"""What is timed when this framework's speed is measured, and over which ranges.

A case is one call a program makes through the public entry points: a host
call of the drop-in module (``kokkos_sim.Component``), the program samplers on
host or device buffers, the device noise draw, the batched launch, a burst of
served requests, or the amplitude evaluation.  Sizes are those of the
repository's own workloads (``ksim_b200.synth``): 5 to 60 outputs, t from 2 to
20 T gates, from a handful to a million shots.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges,
``prepare`` what a program holds before the call, ``run`` one pass of it,
``work`` the bytes and operations a pass cannot do without and ``exact`` the
amplitudes in plain numpy.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from ksim_b200 import _abi, synth
from ksim_b200.batch import BatchSampler
from ksim_b200.kokkos_sim import Component
from ksim_b200.noise import DeviceChannelSampler
from ksim_b200.sampler import B200ProgramSampler
from ksim_b200.serve import Server

_DEV = 0


def listed() -> list:
    return [
        # the drop-in module on a tiny circuit: one interactive call, all latency
        {"name": "component_tiny", "kind": "component", "n_out": 5, "t": 4, "F": 0, "gates": 0, "shots": 64,
         "rng": 0},
        # the small noiseless workload (5 outputs, t = 4) at its own shot count, host arrays
        {"name": "sampler_noiseless", "kind": "sampler", "n_out": 5, "t": 4, "F": 0, "gates": 0,
         "shots": 100_000, "rng": 0},
        # the drop-in module on the 40-output program with numpy arrays, an odd shot count
        {"name": "component_medium", "kind": "component", "n_out": 40, "t": 12, "F": 64, "gates": 200,
         "shots": 20_011, "rng": 0},
        # the 40-output program with inputs and outputs on the device (the headline workload)
        {"name": "device_medium", "kind": "device", "n_out": 40, "t": 12, "F": 64, "gates": 200,
         "shots": 1_000_000, "rng": 0},
        # the large-rank program (16 parity outputs, t = 20), counter-based stream
        {"name": "device_large_rank", "kind": "device", "n_out": 16, "t": 20, "F": 56, "gates": 600,
         "shots": 1_000_000, "rng": 1},
        # few shots of a wide program on the device: a partial wave
        {"name": "device_few_shots", "kind": "device", "n_out": 57, "t": 15, "F": 87, "gates": 570,
         "shots": 3_001, "rng": 0},
        # the 40-output program end to end from page-locked host rows
        {"name": "sampler_pinned", "kind": "pinned", "n_out": 40, "t": 12, "F": 64, "gates": 200,
         "shots": 1_000_000, "rng": 0},
        # noise drawn on the device (8,000 gate locations), outputs to the host
        {"name": "noisy_medium", "kind": "noisy", "n_out": 40, "t": 12, "F": 64, "gates": 200,
         "locations": 8_000, "shots": 300_000, "rng": 0},
        # bit-packed rows of a program of three components with a shuffled output order
        {"name": "packed_multi", "kind": "packed", "specs": "9,22,7;24,40,9;5,11,4", "shots": 77_777, "rng": 1},
        # many programs in one launch: 64 programs, 8 to 60 outputs, t 2 to 16, 1e3 to 1e5 shots
        {"name": "batch_64", "kind": "batch", "programs": 64, "program_seed": 3000, "rng": 0},
        # a burst of requests over a pool of programs through the server
        {"name": "served_burst", "kind": "served", "programs": 16, "requests": 64, "max_shots": 20_000, "rng": 0},
        # amplitudes of one graph for explicit parameter rows (the precision entry point)
        {"name": "eval_abs", "kind": "eval", "n_out": 16, "t": 20, "F": 56, "gates": 600, "graph": 9,
         "shots": 50_000},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["component", "sampler", "device", "device", "pinned", "noisy", "packed", "batch", "served",
                       "eval"])
    if kind == "batch":
        return {"kind": kind, "programs": rng.randint(6, 40), "program_seed": rng.randint(1, 1 << 20), "rng": 0}
    if kind == "served":
        return {"kind": kind, "programs": rng.randint(2, 16), "requests": rng.randint(4, 64),
                "max_shots": _log_int(rng, 500, 20_000), "rng": rng.randint(0, 1)}
    if kind == "packed":
        specs = ";".join("%d,%d,%d" % (rng.randint(2, 24), rng.randint(0, 60), rng.randint(1, 9))
                         for _ in range(rng.randint(1, 3)))
        return {"kind": kind, "specs": specs, "shots": _log_int(rng, 50, 200_000), "rng": rng.randint(0, 1)}
    n_out, t = rng.randint(1, 60), rng.randint(2, 20)
    F = rng.choice([0, n_out, n_out + 2 * t])
    # shots within the cost of the largest listed case (terms x shots)
    terms = (n_out + 1) * max(1.0, 1.1 * 2 ** (0.228 * t))
    top = max(64, int(min(1_000_000, 2.5e8 / terms)))
    case = {"kind": kind, "n_out": n_out, "t": t, "F": F, "gates": rng.choice([100, 200, 10 * n_out]),
            "shots": _log_int(rng, 16, top)}
    if kind == "eval":
        case["graph"] = rng.randint(0, n_out)
        case["shots"] = min(case["shots"], 100_000)
        return case
    case["rng"] = rng.randint(0, 1)
    if kind == "noisy":
        case["F"] = n_out + 2 * t
        case["locations"] = _log_int(rng, 100, 8_000)
        case["shots"] = min(case["shots"], 300_000)
    return case


# ---- the compiled programs (a circuit is compiled once; inputs vary) -------
@functools.lru_cache(maxsize=None)
def _program(n_out: int, t: int, F: int, gates: int):
    """(FlatProgram, f bit probability) of a circuit of this shape."""
    p = synth._noise_prob(gates, F)
    rng = np.random.default_rng(1_000_000 + 10_000 * n_out + 100 * t + F)
    return synth.single_component_program(synth.random_component(rng, n_out=n_out, F=F, t=t, f_prob=p)), p


@functools.lru_cache(maxsize=None)
def _multi_program(specs: str):
    dims = [tuple(int(x) for x in s.split(",")) for s in specs.split(";")]
    return synth.multi_component_program(np.random.default_rng(len(specs) + sum(sum(d) for d in dims)), dims)


@functools.lru_cache(maxsize=None)
def _pool(programs: int):
    return synth.serving_pool(programs)


@functools.lru_cache(maxsize=None)
def _batch(programs: int, seed: int):
    return synth.batched_workloads(programs, seed)


def _rows(seed: int, shots: int, n_f: int, prob: float) -> torch.Tensor:
    """(shots, n_f) uint8 noise bits, Bernoulli(prob), on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.empty((shots, n_f), dtype=torch.uint8, device="cuda")
    if n_f:
        for s in range(0, shots, 1 << 17):
            e = min(shots, s + (1 << 17))
            out[s:e] = torch.rand((e - s, n_f), generator=g, device="cuda") < prob
    return out


def _host_rows(seed: int, shots: int, n_f: int, prob: float) -> np.ndarray:
    return np.ascontiguousarray(_rows(seed, shots, n_f, prob).cpu().numpy())


def _request_shots(case: dict) -> list:
    """Shots of each request of a burst, log-uniform from 100."""
    r = np.random.default_rng(case["requests"])
    return [int(x) for x in np.exp(r.uniform(math.log(100), math.log(case["max_shots"]), case["requests"]))]


def _pinned(shape) -> np.ndarray:
    return torch.zeros(shape, dtype=torch.uint8).pin_memory().numpy()


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"kind": kind, "seed": seed + 17, "rng": int(case.get("rng", 0))}
    if kind == "batch":
        ws = _batch(case["programs"], case["program_seed"])
        bs = BatchSampler([w.program for w in ws], [w.shots for w in ws], seeds=[seed + 31 * i for i in range(len(ws))],
                          rng_mode=st["rng"], device=_DEV, n_f=[w.n_f for w in ws])
        for i, w in enumerate(ws):
            bs.d_f[i].copy_(_rows(seed + 1009 * i, w.shots, w.n_f, w.f_prob))
        return {**st, "batch": bs}
    if kind == "served":
        pool = _pool(case["programs"])
        reqs = []
        for i, b in enumerate(_request_shots(case)):
            w = pool[i % len(pool)]
            f = torch.from_numpy(_host_rows(seed + 7 * i, int(b), w.n_f, w.f_prob)).pin_memory().numpy()
            reqs.append((w.program, f, seed + i, _pinned((int(b), w.program.num_outputs))))
        srv = Server(device=_DEV, arena_bytes=1 << 28)
        for w in pool:  # programs resident before the stream
            srv.cache.release(srv.cache.acquire(w.program)[0])
        return {**st, "server": srv, "requests": reqs}
    shots = case["shots"]
    if kind == "packed":
        prog, n_f = _multi_program(case["specs"])
        f = np.packbits(_host_rows(seed, shots, n_f, 0.02), axis=1, bitorder="little")
        s = B200ProgramSampler(prog, device=_DEV)
        out = _pinned((shots, (s.num_outputs + 7) // 8))
        return {**st, "sampler": s, "n_f": n_f, "out": out, "f": torch.from_numpy(f).pin_memory().numpy()}
    prog, p = _program(case["n_out"], case["t"], case["F"], case["gates"])
    if kind == "eval":
        comp = Component(prog.components[0].graphs, case["F"], device=_DEV)
        return {**st, "component": comp, "graph": case["graph"], "params": _params(case, seed)}
    if kind == "component":
        comp = Component(prog.components[0].graphs, case["F"], device=_DEV)
        return {**st, "component": comp, "f": _host_rows(seed, shots, case["F"], p)}
    s = B200ProgramSampler(prog, device=_DEV)
    if kind == "device":
        return {**st, "sampler": s, "f": _rows(seed, shots, case["F"], p),
                "out": torch.zeros((shots, s.num_outputs), dtype=torch.uint8, device="cuda")}
    if kind == "noisy":
        probs, T = synth.noise_model(np.random.default_rng(seed), case["F"], case["locations"])
        return {**st, "sampler": s, "noise": DeviceChannelSampler(probs, T, seed=seed, device=_DEV), "shots": shots,
                "out": _pinned((shots, s.num_outputs))}
    f = _host_rows(seed, shots, case["F"], p)
    if kind == "pinned":
        return {**st, "sampler": s, "f": torch.from_numpy(f).pin_memory().numpy() if f.size else f,
                "out": _pinned((shots, s.num_outputs))}
    return {**st, "sampler": s, "f": f}


def run(st: dict):
    kind = st["kind"]
    if kind == "component":
        return st["component"].sample(st["f"], st["seed"], rng_mode=st["rng"])
    if kind == "sampler":
        return st["sampler"].sample(st["f"], st["seed"], rng_mode=st["rng"])
    if kind == "pinned":
        return st["sampler"].sample(st["f"], st["seed"], rng_mode=st["rng"], out=st["out"])
    if kind == "packed":
        return st["sampler"].sample_packed(st["f"], st["n_f"], st["seed"], rng_mode=st["rng"], out=st["out"])
    if kind == "noisy":
        return st["sampler"].sample_noisy(st["noise"], st["shots"], st["seed"], rng_mode=st["rng"], out=st["out"])
    if kind == "device":
        f, out = st["f"], st["out"]
        _abi.check(_abi.lib().ksim_program_sample_device(
            st["sampler"].handle, ctypes.c_void_p(f.data_ptr()), f.shape[0], f.shape[1], 0, st["seed"], st["rng"],
            ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return out
    if kind == "batch":
        st["batch"].launch()
        return list(st["batch"].d_out)
    if kind == "served":
        hs = [st["server"].submit(prog, f, seed, st["rng"], out=out) for prog, f, seed, out in st["requests"]]
        return [h.result() for h in hs]
    return st["component"].eval_abs(st["graph"], st["params"])


# ---- what a pass cannot do without ------------------------------------------
@functools.lru_cache(maxsize=None)
def _program_work(key: tuple) -> tuple:
    """(operations of one shot, bytes of its input and output row)."""
    if key[0] == "multi":
        prog, n_f = _multi_program(key[1])
    else:
        prog, n_f = _program(*key[1:])[0], key[3]
    return _ops(prog), n_f + prog.num_outputs


def _ops(prog, graph=None) -> float:
    """One operation per mask of a term's columns and two additions per term."""
    ops = 0.0
    for c in prog.components:
        for k, g in enumerate(c.graphs):
            if graph is None or k == graph:
                G = g.pf_phase_idx.shape[0]
                ops += float(np.maximum(g.np_counts, 0).sum() + 2 * np.maximum(g.ph_counts, 0).sum())
                ops += G * (g.hp_coeffs.shape[1] + 2 * g.pp_psi_c.shape[1] + 2)
    return ops


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        ws = _batch(case["programs"], case["program_seed"])
        return {"bytes": float(sum(w.shots * (w.n_f + w.program.num_outputs) for w in ws)),
                "flops": float(sum(w.shots * _ops(w.program) for w in ws))}
    if kind == "served":
        pool = _pool(case["programs"])
        use = [(b, pool[i % len(pool)]) for i, b in enumerate(_request_shots(case))]
        return {"bytes": float(sum(b * (w.n_f + w.program.num_outputs) for b, w in use)),
                "flops": float(sum(b * _ops(w.program) for b, w in use))}
    shots = case["shots"]
    if kind == "eval":
        prog, _ = _program(case["n_out"], case["t"], case["F"], case["gates"])
        return {"bytes": float(shots * (case["F"] + case["graph"] + 8)),
                "flops": float(shots * _ops(prog, case["graph"]))}
    if kind == "packed":
        ops, row = _program_work(("multi", case["specs"]))
        return {"bytes": float(shots * row / 8), "flops": float(shots * ops)}
    ops, row = _program_work(("one", case["n_out"], case["t"], case["F"], case["gates"]))
    if kind == "noisy":
        row -= case["F"]  # f never leaves the device
    return {"bytes": float(shots * row), "flops": float(shots * ops)}


# ---- amplitudes in plain numpy ----------------------------------------------
def _params(case: dict, seed: int) -> np.ndarray:
    """Parameter rows of the evaluation case: f bits, sampled bits, the trying bit."""
    prog, p = _program(case["n_out"], case["t"], case["F"], case["gates"])
    P = prog.components[0].graphs[case["graph"]].np_params.shape[2]
    r = np.random.default_rng(seed)
    rows = (r.random((case["shots"], P)) < 0.5).astype(np.uint8)
    rows[:, :case["F"]] = r.random((case["shots"], case["F"])) < max(p, 0.05)
    if case["graph"] > 0:
        rows[:, P - 1] = 1
    return rows


def exact(case: dict, seed: int):
    """|A| of each parameter row in 64 bits: a sum over the graph's terms of
    products of cyclotomic factors selected by parities.  The sampled bits of
    the other cases are whole numbers."""
    if case["kind"] != "eval":
        return None
    g = _program(case["n_out"], case["t"], case["F"], case["gates"])[0].components[0].graphs[case["graph"]]
    x = _params(case, seed).astype(np.float64)
    unit = np.exp(1j * np.pi / 4 * np.arange(8))
    total = np.zeros(x.shape[0], complex)

    def parity(m):
        if m.shape[0] == 0:
            return np.zeros((x.shape[0], 0), np.int64)
        return (x[:, :m.shape[1]] @ m.astype(np.float64).T).astype(np.int64) & 1

    for t in range(g.pf_phase_idx.shape[0]):
        n, m = max(0, int(g.np_counts[t])), max(0, int(g.ph_counts[t]))
        z = (1 + unit[(4 * parity(g.np_params[t, :n]) + g.np_phases[t, :n]) & 7]).prod(axis=1)
        k = (parity(g.hp_params[t]) * g.hp_coeffs[t]).sum(axis=1)
        k = k + 4 * (((parity(g.pp_psi_p[t]) + g.pp_psi_c[t]) & 1) * ((parity(g.pp_phi_p[t]) + g.pp_phi_c[t]) & 1)).sum(axis=1)
        a = (4 * parity(g.ph_alpha_p[t, :m]) + g.ph_alpha[t, :m]) & 7
        b = (4 * parity(g.ph_beta_p[t, :m]) + g.ph_beta[t, :m]) & 7
        z = z * (1 + unit[a] + unit[b] - unit[(a + b) & 7]).prod(axis=1)
        ff = g.pf_floatfactor[t].astype(float)
        z = z * unit[(k + int(g.pf_phase_idx[t])) & 7] * (ff[0] + ff[1] * unit[1] + ff[2] * 1j + ff[3] * np.conj(unit[1]))
        z = z * 2.0 ** float(g.pf_power2[t])
        total += z * (complex(g.pf_approx[t]) if g.pf_has_approx else 1.0)
    return np.abs(total)
