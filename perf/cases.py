"""Performance cases of the population-annealing engine: what its users have it do, through its public
entry points (paising_gb300.Engine and paising_gb300.stages).

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call: an engine handle, or device tensors
    run(state)           one pass, and its outputs
    work(case)           bytes and integer operations a pass cannot do without
    exact(case, seed)    the outputs in 64 bits, where they are computed numbers

Whole anneals dominate: the engine's work is the temperature loop, so its kernels (sweep, resampling plan,
gather, bookkeeping) run at the proportions a user's anneal gives them.  The stage cases are the calls of a
program that drives the temperature loop itself on its own device buffers.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import paising_gb300 as pa
from paising_gb300 import stages


# ------------------------------------------------------------------ the cases
def _anneal(**kw) -> dict:
    c = dict(kind="anneal", L=64, R=20000, sweeps=100, dbeta=0.005, coding="msc", runs=1, weights="fp32",
             adaptive=False, mhr=False, family=False)
    c.update(kw)
    return c


def listed() -> list[dict]:
    return [
        # the smallest production anneal: 199 temperatures of a 16 x 16 lattice, a few microseconds of spin
        # flips each, so launches and the per-temperature kernels' latency are what a user waits for
        _anneal(name="anneal_ssc_L16_R1000", coding="ssc", L=16, R=1000, sweeps=10),
        # the reference's sample shape (L = 64, R = 20000, 100 sweeps, dbeta = 0.005), one population, MSC
        _anneal(name="anneal_msc_L64_R20000"),
        # the same shape in single-spin coding, with a coarser schedule
        _anneal(name="anneal_ssc_L64_R20000", coding="ssc", dbeta=0.02),
        # independent runs of that shape annealed together (the reference's -M 8), with a coarser schedule
        _anneal(name="anneal_msc_L64_R20000_runs8", dbeta=0.02, runs=8),
        # a large lattice: a group of 32 replicas does not fit one thread block's shared memory
        _anneal(name="anneal_msc_L256_R8192", L=256, R=8192, sweeps=50, dbeta=0.05),
        # a large population with few sweeps per temperature and strong reweighting, all-FP64 weights (the
        # precision study's L = 32, R = 10^6): resampling weighs as much as the sweeps
        _anneal(name="anneal_msc_L32_R1000000_fp64", L=32, R=1_000_000, sweeps=5, dbeta=0.05, weights="fp64"),
        # the reference's adaptive temperature step with multi-histogram reweighting and family statistics
        _anneal(name="anneal_msc_L32_R5000_adaptive", L=32, R=5000, sweeps=20, adaptive=True, mhr=True, family=True),
        # populations of uneven lattice and population sizes and schedules annealed as one batch
        dict(kind="batch", name="batch_msc_uneven16", coding="msc", npop=16, pick=2026, Rmin=1000, Rmax=8000,
             sweeps=20),
        # the resampling plan of one temperature (weights, copy numbers, scan, gather map), MSC, ragged last group
        dict(kind="plan", name="plan_msc_R20001", coding="msc", R=20001, spread=0.3, weights="fp32"),
        # the gather of the resampled population, MSC: a population larger than L2
        dict(kind="gather", name="gather_msc_L128_R131072", coding="msc", L=128, R=131072, spread=0.3),
        # the gather of the resampled population, SSC int8
        dict(kind="gather", name="gather_ssc_L64_R100000", coding="ssc", L=64, R=100000, spread=0.3),
        # the int8 sweep, of the lattice sizes without a dense bit-plane layout: L = 40, odd replica count
        dict(kind="sweep", name="sweep_ssc_L40_R3001", form="ssc", L=40, R=3001, sweeps=20, beta=0.44),
    ]


# spin-flip attempts of the largest drawn case (the listed single-population MSC anneal makes 1.6e12)
_MAX_ATTEMPTS = 1.2e12


def _log_int(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["anneal", "anneal", "anneal", "batch", "plan", "gather", "sweep"])
    if kind == "anneal":
        coding = rng.choice(["msc", "msc", "ssc"])
        L = rng.choice([8, 16, 24, 32, 40, 48, 64, 64, 72, 96, 128, 160, 192, 256]) if coding == "ssc" else \
            rng.choice([10, 12, 16, 20, 32, 36, 48, 64, 64, 70, 96, 100, 128, 144, 192, 256])
        sweeps = _log_int(rng, 5, 100)
        dbeta = rng.choice([0.005, 0.01, 0.02, 0.05])
        runs = rng.choice([1, 1, 1, 2, 5])
        per = sweeps * L * L * runs / dbeta
        if coding == "ssc":
            per *= 6  # the int8 sweep of the sizes without a dense bit-plane layout makes fewer attempts per second
        R = _log_int(rng, 300, max(600.0, min(500_000.0 / runs, _MAX_ATTEMPTS / per)))
        adaptive = rng.random() < 0.15
        return _anneal(coding=coding, L=L, R=R, sweeps=sweeps, dbeta=dbeta, runs=1 if adaptive else runs,
                       weights=rng.choice(["fp32", "fp32", "fp64"]), adaptive=adaptive, mhr=rng.random() < 0.2,
                       family=rng.random() < 0.2)
    if kind == "batch":
        return dict(kind="batch", coding=rng.choice(["msc", "ssc"]), npop=rng.randint(3, 24), pick=rng.randint(0, 10**6),
                    Rmin=rng.randint(300, 1000), Rmax=rng.randint(2000, 6000), sweeps=rng.randint(5, 20))
    if kind == "plan":
        return dict(kind="plan", coding=rng.choice(["msc", "ssc"]), R=_log_int(rng, 1000, 1_000_000),
                    spread=rng.choice([0.05, 0.3, 1.0]), weights=rng.choice(["fp32", "fp32", "fp64"]))
    if kind == "gather":
        coding = rng.choice(["msc", "ssc"])
        L = rng.choice([16, 32, 40, 64, 96, 128, 256] if coding == "ssc" else [10, 16, 30, 32, 64, 96, 128, 256])
        top = 6e8 / (L * L) if coding == "ssc" else 2.4e9 / (L * L)
        return dict(kind="gather", coding=coding, L=L, R=_log_int(rng, 1000, min(1_000_000.0, top)),
                    spread=rng.choice([0.05, 0.3, 1.0]))
    form = rng.choice(["ssc", "ssc_bits", "msc"])
    L = rng.choice({"ssc": [8, 16, 40, 64, 72, 128], "ssc_bits": [16, 24, 32, 64, 96, 128, 192],
                    "msc": [10, 16, 30, 48, 64, 96, 100, 128]}[form])
    sweeps = _log_int(rng, 5, 100)
    return dict(kind="sweep", form=form, L=L, R=_log_int(rng, 500, min(200_000.0, 5e10 / (sweeps * L * L))), sweeps=sweeps,
                beta=round(rng.uniform(0.05, 1.0), 3))


# ------------------------------------------------------------- their inputs
def _batch_pops(case: dict, seed: int) -> list[dict]:
    """The batch's populations: L, R, dbeta from the case's pick alone, their seeds from `seed`."""
    r = random.Random(case["pick"])
    return [dict(L=r.choice([16, 32, 48, 64, 96, 128]), R=r.randint(case["Rmin"], case["Rmax"]),
                 dbeta=r.choice([0.01, 0.02, 0.05]), sweeps=case["sweeps"], seed=1000 * seed + k)
            for k in range(case["npop"])]


def _energies(case: dict, gen: torch.Generator) -> torch.Tensor:
    """Energies of R replicas as an L = 64 population near the transition has them: multiples of 4, spread so
    that dbeta times the standard deviation is the case's `spread` at dbeta = 0.005."""
    sd = case["spread"] / 0.005
    e = torch.randn(case["R"], generator=gen, device="cuda", dtype=torch.float64) * sd - 5800.0
    return (4.0 * torch.round(e / 4.0)).clamp(-8192, 0).to(torch.int32)


def _source_map(case: dict, gen: torch.Generator) -> torch.Tensor:
    """New replica -> old replica, nondecreasing: systematic resampling of R replicas with log-normal weights of
    the case's spread (copy numbers within one of their expectation, as the engine's are)."""
    x = torch.randn(case["R"], generator=gen, device="cuda", dtype=torch.float64) * case["spread"]
    edge = torch.softmax(x, 0).cumsum(0) * case["R"]
    at = torch.arange(case["R"], device="cuda", dtype=torch.float64) + float(torch.rand((), generator=gen, device="cuda"))
    return torch.searchsorted(edge, at, right=True).clamp(max=case["R"] - 1).to(torch.int32)


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "anneal":
        keys = ("L", "R", "sweeps", "dbeta", "coding", "runs", "weights", "adaptive", "mhr", "family")
        # a strongly reweighted small population can outgrow the default replica buffer
        N, R = case["L"] ** 2, case["R"]
        # the final population beside the rows, where a program would fetch it: up to 16 MB
        fetch = case["runs"] == 1 and R * N // (8 if case["coding"] == "msc" else 1) <= 2**24
        return {"kind": kind, "runs": case["runs"], "mhr": case["mhr"], "family": case["family"],
                "adaptive": case["adaptive"], "slots": R + R // 2 + 512 if fetch else 0,
                "engine": pa.Engine(seed=seed, capacity=1.5, **{k: case[k] for k in keys})}
    if kind == "batch":
        return {"kind": kind, "npop": case["npop"],
                "engine": pa.Engine.batch(_batch_pops(case, seed), coding=case["coding"], capacity=1.5)}
    R = case["R"]
    if kind == "plan":
        E = _energies(case, gen)
        st = {"kind": kind, "R": R, "weights": pa.WEIGHTS_FP64 if case["weights"] == "fp64" else pa.WEIGHTS_FP32,
              "coding": pa.MSC if case["coding"] == "msc" else pa.SSC, "active": None, "seed": seed,
              "e_ref": float(E.double().mean()) if case["weights"] == "fp64" else float(E.min())}
        if case["coding"] == "msc":  # whole groups of 32 slots, the last one partly active
            n = (R + 31) // 32 * 32
            st["active"] = (torch.arange(n, device="cuda") < R).to(torch.uint8)
            E = torch.cat([E, torch.zeros(n - R, dtype=torch.int32, device="cuda")])
        st["E"] = E
        return st
    if kind == "gather":
        L = case["L"]
        src = _source_map(case, gen)
        if case["coding"] == "msc":
            old = torch.randint(-2**31, 2**31, ((R + 31) // 32, L * L), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
        else:
            old = torch.randint(0, 2, (R, L * L), generator=gen, device="cuda", dtype=torch.int8) * 2 - 1
        return {"kind": kind, "coding": case["coding"], "L": L, "R": R, "src": src, "R_new": src.shape[0], "old": old}
    # sweep: a population half-way ordered, as a warm anneal has it (each site +1 with probability 0.8)
    L = case["L"]
    st = {"kind": kind, "form": case["form"], "L": L, "sweeps": case["sweeps"], "beta": case["beta"], "seed": seed}
    if case["form"] == "msc":
        rg = (R + 31) // 32
        w = torch.zeros((rg, L * L), dtype=torch.int32, device="cuda")
        for b in range(32):
            bit = (torch.rand((rg, L * L), generator=gen, device="cuda") < 0.8).to(torch.int32)
            w |= bit << b
        st["words"] = w
        st["active"] = (torch.arange(rg * 32, device="cuda") < R).to(torch.uint8)
    else:
        st["spins"] = (torch.rand((R, L * L), generator=gen, device="cuda") < 0.8).to(torch.int8) * 2 - 1
    return st


# -------------------------------------------------------------------- a pass
def _table(rows: np.ndarray, adaptive: bool) -> np.ndarray:
    """A result table; of an adaptive run, whose length is the run's own, in a block of 1024 rows."""
    if not adaptive:
        return rows
    out = np.zeros((1024, rows.shape[1]))
    out[: len(rows)] = rows
    return out


def _whole(pop: np.ndarray, slots: int) -> np.ndarray:
    """The population's replicas (its size is the run's own) at the head of a block of `slots` replicas."""
    n = slots if pop.dtype == np.int8 else slots // 32
    out = np.zeros((n, pop.shape[1]), dtype=np.int8 if pop.dtype == np.int8 else np.int32)
    out[: len(pop)] = pop.view(out.dtype)
    return out


def run(state: dict):
    kind = state["kind"]
    if kind == "anneal":
        e, ad = state["engine"], state["adaptive"]
        e.run()
        out = {"rows": [_table(e.rows(k), ad) for k in range(state["runs"])]}
        if state["slots"]:
            out["population"] = _whole(e.population(), state["slots"])
        if state["mhr"]:
            out["mhr"] = [_table(e.mhr_rows(k), ad) for k in range(state["runs"])]
        if state["family"]:
            out["family"] = [_table(e.family_rows(k), ad) for k in range(state["runs"])]
        return out
    if kind == "batch":
        e = state["engine"]
        e.run()
        return {"rows": [e.rows(k) for k in range(state["npop"])]}
    if kind == "plan":
        R = state["R"]
        roff, offs, src, lnq, q, rn = stages.resample_plan(state["E"], state["active"], state["coding"], R, R,
                                                           R + R // 4 + 256, 0.44, 0.445, state["e_ref"],
                                                           state["weights"], state["seed"], 12345)
        src[rn:].zero_()  # the map is written for the new population's replicas; the rest of the buffer is spare
        return {"copies": roff, "offsets": offs, "src": src, "lnQ": lnq, "q": q, "R": rn}
    if kind == "gather":
        if state["coding"] == "msc":
            new, act = stages.msc_resample_native(state["old"], state["L"], state["R"], state["src"], state["R_new"])
            return {"new": new, "active": act}
        return {"new": stages.ssc_resample(state["old"], state["L"], state["src"], state["R_new"])}
    L, n, beta, seed = state["L"], state["sweeps"], state["beta"], state["seed"]
    if state["form"] == "msc":
        E, M = stages.msc_sweep(state["words"], state["active"], L, n, beta, pa.RNG_NATIVE, seed)
        return {"spins": state["words"], "E": E, "M": M}
    if state["form"] == "ssc":
        E, M = stages.ssc_sweep(state["spins"], L, n, beta, pa.RNG_NATIVE, seed)
    else:
        E, M = stages.ssc_sweep_bits(state["spins"], L, n, beta, seed)
    return {"spins": state["spins"], "E": E, "M": M}


# ---------------------------------------------------------------------- work
# Integer operations of one spin-flip attempt: multi-spin coding (and bit planes, which share its machinery)
# neighbour counts, random bits and decisions of 32 spins per word; int8 single-spin coding, one site at a time.
_OPS_WORD, _OPS_INT8 = 5, 33
_DENSE = {8, 16, 24, 32, 48, 56, 64, 96, 112, 128, 144, 168, 192, 224, 240, 256}  # SSC sizes swept on bit planes


def _steps(dbeta: float) -> int:
    b, n = 0.0, 0  # beta accumulated up to 1, as the schedule is
    while b + dbeta <= 1.0:
        b, n = b + dbeta, n + 1
    return n


def _anneal_work(coding: str, L: int, R: int, sweeps: int, steps: int) -> tuple[float, float]:
    attempts = float(sweeps) * L * L * R * steps
    ops = _OPS_WORD if coding == "msc" or L in _DENSE else _OPS_INT8
    state = R * L * L / 8 if coding == "msc" else float(R) * L * L
    # per temperature: the population is read and rewritten (sweep with the gather folded in), energies too
    return steps * (2 * state + 8.0 * R), attempts * ops


def work(case: dict) -> dict:
    kind = case["kind"]
    R = case.get("R", 0)
    if kind == "anneal":
        # the adaptive step's length is the run's own: about 1.5 sqrt(N) temperatures at overlaps of 0.85 .. 0.87
        steps = int(1.5 * case["L"]) if case["adaptive"] else _steps(case["dbeta"])
        b, f = _anneal_work(case["coding"], case["L"], R * case["runs"], case["sweeps"], steps)
        return {"bytes": b, "flops": f}
    if kind == "batch":
        w = [_anneal_work(case["coding"], p["L"], p["R"], p["sweeps"], _steps(p["dbeta"])) for p in _batch_pops(case, 0)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    if kind == "plan":  # energies (and active flags) read; copy numbers, offsets and the map written
        return {"bytes": R * (4.0 + 12.0 + (1.0 if case["coding"] == "msc" else 0.0)), "flops": 60.0 * R}
    if kind == "gather":
        per = case["L"] ** 2 / (8.0 if case["coding"] == "msc" else 1.0)
        return {"bytes": R * (2 * per + 4.0), "flops": 0.0}
    per = case["L"] ** 2 / (8.0 if case["form"] == "msc" else 1.0)
    ops = _OPS_INT8 if case["form"] == "ssc" else _OPS_WORD
    return {"bytes": R * (2 * per + 8.0), "flops": float(case["sweeps"]) * case["L"] ** 2 * R * ops}


# --------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    """The resampling plan's lnQ and q in 64 bits.  Every other output is a whole number or a byte (spins,
    energies, copy numbers), or a row of an anneal, which follows from the engine's own random stream."""
    if case["kind"] != "plan":
        return None
    gen = torch.Generator(device="cuda").manual_seed(seed)
    E = _energies(case, gen).cpu().numpy().astype(np.float64)
    e_ref = float(E.mean()) if case["weights"] == "fp64" else float(E.min())
    db = 0.445 - 0.44
    q = float(np.sum(np.exp(-db * (E - e_ref)).astype(np.longdouble)))
    return {"copies": None, "offsets": None, "src": None, "lnQ": -db * e_ref + math.log(q) - math.log(len(E)),
            "q": q, "R": None}
