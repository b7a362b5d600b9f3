"""The annealing work that a user of this framework has it do, as timed cases.

Each case is one call of a public entry point: the C ABI's annealing runs (through its ctypes view, spins and
energies in device memory, on torch's current stream), or a whole sampler call.  A pass sets the replicas to the
caller's start states, anneals them over a whole schedule and returns every replica's spins and FP64 energies.
The instances are the families of openjij_b200/instances.py, drawn from the seed; the sizes are those of the
benchmark's workloads and of the tests, with ragged ones beside them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from openjij_b200 import _native as N
from openjij_b200 import instances as I


def listed():
    return [
        # a small dense Ising problem annealed by 100 reads, the benchmark's smallest workload
        {"name": "sa dense n=100 real", "kind": "sa", "family": "dense_real", "n": 100, "R": 100, "S": 1000,
         "b0": 0.1, "b1": 10.0},
        # an ordinary dense QUBO with real coefficients, ragged in sites and reads
        {"name": "sa dense n=777 real", "kind": "sa", "family": "dense_real", "n": 777, "R": 200, "S": 500,
         "b0": 0.1, "b1": 10.0},
        # the benchmark's large integer QUBO with 4096 replicas
        {"name": "sa dense n=2048 int", "kind": "sa", "family": "dense_int", "n": 2048, "R": 4096, "S": 1000,
         "b0": 0.05, "b1": 5.0},
        # the +-J spin glass of the default benchmark line: one regular lattice, many replicas, a long schedule
        {"name": "sa lattice L=128", "kind": "sa", "family": "lattice", "n": 128, "R": 1024, "S": 2000,
         "b0": 0.1, "b1": 5.0},
        # the same model at an odd side (not bipartite) with a replica count that fills no word
        {"name": "sa lattice L=33", "kind": "sa", "family": "lattice", "n": 33, "R": 100, "S": 1000,
         "b0": 0.1, "b1": 5.0},
        # an annealer's Chimera graph with real fields: the sparse path for anything that is not a pure +-J lattice
        {"name": "sa chimera L=16 fields", "kind": "sa", "family": "chimera", "n": 16, "R": 1024, "S": 1000,
         "b0": 0.1, "b1": 5.0},
        # many dense QUBOs of uneven size in one call
        {"name": "sa batch 64 x n<=512", "kind": "batch", "count": 64, "nmin": 64, "nmax": 512, "R": 32, "S": 500,
         "b0": 0.1, "b1": 10.0},
        # simulated quantum annealing of a 3-regular spin glass with 32 Trotter slices, the benchmark's workload
        {"name": "sqa 3-regular n=4096 T=32", "kind": "sqa", "family": "regular", "n": 4096, "T": 32, "R": 256,
         "S": 1000, "beta": 10.0},
        # SQASampler's defaults (4 slices, beta 5, 1000 sweeps) on a dense QUBO with real coefficients
        {"name": "sqa dense n=64 T=4", "kind": "sqa", "family": "dense_real", "n": 64, "T": 4, "R": 100, "S": 1000,
         "beta": 5.0},
        # SQA on a Chimera graph with real fields
        {"name": "sqa chimera L=8 T=8", "kind": "sqa", "family": "chimera", "n": 8, "T": 8, "R": 128, "S": 500,
         "beta": 5.0},
        # the cluster updater on the lattice where single flips freeze
        {"name": "swendsen-wang lattice L=64", "kind": "sw", "family": "lattice", "n": 64, "R": 256, "S": 200,
         "b0": 0.1, "b1": 5.0},
        # a whole sampler call on a small QUBO dictionary with the sampler's own schedule: call overhead
        {"name": "sampler qubo n=24", "kind": "sampler", "n": 24, "R": 10, "S": 1000},
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["dense_small", "dense_real", "dense_int", "lattice", "chimera", "batch", "sqa_regular",
                       "sqa_dense", "sqa_chimera", "sw", "sampler"])
    if kind == "dense_small":
        return {"kind": "sa", "family": rng.choice(["dense_real", "dense_int"]), "n": _spread(rng, 5, 128),
                "R": _spread(rng, 1, 1000), "S": _spread(rng, 100, 1000), "b0": 0.1, "b1": 10.0}
    if kind == "dense_real":
        return {"kind": "sa", "family": "dense_real", "n": _spread(rng, 129, 1500), "R": _spread(rng, 1, 512),
                "S": _spread(rng, 50, 500), "b0": 0.1, "b1": 10.0}
    if kind == "dense_int":
        return {"kind": "sa", "family": "dense_int", "n": _spread(rng, 129, 2048), "R": _spread(rng, 1, 4096),
                "S": _spread(rng, 100, 1000), "b0": 0.05, "b1": 5.0}
    if kind == "lattice":
        return {"kind": "sa", "family": "lattice", "n": _spread(rng, 6, 128), "R": _spread(rng, 1, 1024),
                "S": _spread(rng, 100, 2000), "b0": 0.1, "b1": 5.0}
    if kind == "chimera":
        return {"kind": "sa", "family": "chimera", "n": _spread(rng, 2, 24), "R": _spread(rng, 1, 1024),
                "S": _spread(rng, 100, 1000), "b0": 0.1, "b1": 5.0}
    if kind == "batch":
        nmin = _spread(rng, 16, 128)
        return {"kind": "batch", "count": _spread(rng, 2, 64), "nmin": nmin, "nmax": _spread(rng, nmin, 512),
                "R": _spread(rng, 1, 64), "S": _spread(rng, 50, 500), "b0": 0.1, "b1": 10.0}
    if kind == "sqa_regular":
        return {"kind": "sqa", "family": "regular", "n": 2 * _spread(rng, 32, 2048),
                "T": rng.choice([4, 5, 8, 10, 16, 32]), "R": _spread(rng, 1, 256), "S": _spread(rng, 100, 1000),
                "beta": 10.0}
    if kind == "sqa_dense":
        T = rng.choice([2, 4, 5, 8, 16])
        return {"kind": "sqa", "family": rng.choice(["dense_real", "dense_int"]), "n": _spread(rng, 5, 64), "T": T,
                "R": _spread(rng, 1, 100), "S": _spread(rng, 100, 1000 if T <= 4 else 400), "beta": 5.0}
    if kind == "sqa_chimera":
        return {"kind": "sqa", "family": "chimera", "n": _spread(rng, 2, 12), "T": rng.choice([2, 4, 7, 8, 16]),
                "R": _spread(rng, 1, 128), "S": _spread(rng, 100, 500), "beta": 5.0}
    if kind == "sw":
        return {"kind": "sw", "family": rng.choice(["lattice", "chimera"]), "n": _spread(rng, 4, 20)
                if rng.random() < 0.5 else _spread(rng, 6, 24), "R": _spread(rng, 1, 256),
                "S": _spread(rng, 50, 200), "b0": 0.1, "b1": 5.0}
    return {"kind": "sampler", "n": _spread(rng, 3, 100), "R": _spread(rng, 1, 100), "S": _spread(rng, 100, 1000)}


def _instance(case, seed):
    """The symmetric augmented matrix of a case's instance."""
    family, n = case["family"], case["n"]
    if family == "dense_real":
        return I.dense_ising_uniform(n, seed=seed)[0]
    if family == "dense_int":
        return I.dense_qubo_int(n, seed=seed)[0]
    if family == "lattice":
        return I.lattice_pm_j(n, seed=seed)[0]
    if family == "chimera":
        return I.chimera_pm_j(n, seed=seed, field=0.5)[0]
    return I.random_regular_pm_j(n, 3, seed=seed)[0]


def _sites(case):
    if case.get("family") == "lattice":
        return case["n"] ** 2
    if case.get("family") == "chimera":
        return 8 * case["n"] ** 2
    return case["n"]


def _couplings(case):
    """Couplings of a case's instance, each pair once."""
    n = case["n"]
    return {"lattice": 2 * n * n, "chimera": 16 * n * n + 8 * n * (n - 1), "regular": 3 * n // 2}.get(
        case.get("family"), n * (n - 1) // 2)


def _batch_sizes(case):
    return np.random.default_rng(case["count"]).integers(case["nmin"], case["nmax"] + 1, size=case["count"])


def _random_spins(shape, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randint(0, 2, shape, generator=gen, device="cuda", dtype=torch.int8) * 2 - 1).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "seed": seed}
    if kind == "sampler":
        from openjij_b200.sampler import sa_sampler
        rng = np.random.default_rng(seed)
        n = case["n"]
        q = np.round(rng.uniform(-1.0, 1.0, size=(n, n)), 3)
        state["Q"] = {(i, j): float(q[i, j]) for i in range(n) for j in range(i, n)}
        state["sampler"] = sa_sampler.SASampler()
        return state
    ctx = N.Context(torch.cuda.current_device())
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    state["ctx"] = ctx
    S = case["S"]
    if kind == "batch":
        sizes = _batch_sizes(case)
        state["plan"] = N.Batch(ctx, [I.dense_qubo_normal(int(n), seed * 1009 + k)[0].toarray()
                                      for k, n in enumerate(sizes)])
        state["reads"] = np.full(len(sizes), case["R"], np.int32)
        shape, count = (int(sizes.sum()) * case["R"],), len(sizes) * case["R"]
    else:
        state["plan"] = N.Graph(ctx, *I.augmented_csr(_instance(case, seed)))
        n = _sites(case)
        shape = (case["R"], case["T"], n) if kind == "sqa" else (case["R"], n)
        count = case["R"] * case.get("T", 1)
    if kind == "sqa":
        # SQASampler's schedule: fixed beta, s along the quartic curve from 0 to 1
        x = np.linspace(0.0, 1.0, S)
        state["betas"], state["mcs"] = np.full(S, case["beta"]), np.ones(S, np.int32)
        state["s"] = x**4 * (35 - 84 * x + 70 * x**2 - 20 * x**3)
        state["best"] = torch.zeros(case["R"], dtype=torch.int32, device="cuda")
    else:
        state["betas"], state["mcs"] = I.geometric_betas(case["b0"], case["b1"], S)
    state["start"] = _random_spins(shape, seed)
    state["spins"] = torch.empty_like(state["start"])
    state["energies"] = torch.zeros(count, dtype=torch.float64, device="cuda")
    return state


def run(state):
    kind, case, seed = state["case"]["kind"], state["case"], state["seed"]
    if kind == "sampler":
        r = state["sampler"].sample_qubo(state["Q"], num_reads=case["R"], num_sweeps=case["S"], seed=seed)
        return {"states": r.states, "energies": r.energies}
    spins, energies = state["spins"], state["energies"]
    spins.copy_(state["start"])
    out = {"spins": spins, "energies": energies}
    if kind == "batch":
        N.sa_run_batched(state["plan"], state["reads"], spins, state["betas"], state["mcs"], seed,
                         energies=energies, device=True)
    elif kind == "sqa":
        N.sqa_run(state["plan"], spins, 1.0, state["betas"], state["s"], state["mcs"], seed, energies=energies,
                  best=state["best"], device=True)
        out["best"] = state["best"]
    elif kind == "sw":
        N.sw_run(state["plan"], spins, state["betas"], state["mcs"], seed, energies=energies, device=True)
    else:
        N.sa_run(state["plan"], spins, state["betas"], state["mcs"], seed, energies=energies, device=True)
    return out


def work(case):
    """Bytes: couplings, fields and start states in, spins and energies out, once.  Operations: one acceptance test
    (product with beta, logarithm of the uniform, comparison) per attempt, and the field's additions: one per
    neighbour of a sparse site; a dense site's field follows the accepted flips, counted as one in a hundred."""
    kind, R, S, T = case["kind"], case["R"], case["S"], case.get("T", 1)
    if kind == "batch":
        n = (case["nmin"] + case["nmax"]) / 2.0
        n2 = (case["nmax"] ** 2 + case["nmin"] * case["nmax"] + case["nmin"] ** 2) / 3.0
        return {"bytes": case["count"] * (4.0 * n2 + 4.0 * n + 2.0 * R * n + 8.0 * R),
                "flops": case["count"] * float(R) * S * (3.0 * n + 0.02 * n2)}
    n, m = _sites(case), _couplings(case)
    dense = kind == "sampler" or case["family"].startswith("dense")
    per = 3.0 + (0.02 * n if dense else 2.0 * m / n)
    return {"bytes": 8.0 * m + 4.0 * n + 2.0 * R * T * n + 8.0 * R * T, "flops": per * R * T * n * float(S)}


def exact(case, seed):
    """None: the energies are those of the spins that a case's random walk ends in."""
    return None
