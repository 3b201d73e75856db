"""Performance cases: what users of this package have it do, through its public entry points.

Five kinds of pass, each from small to large and at odd sizes:

``election``  ballots on the GPU through tally, strongest paths and ranking: one whole Schulze
              election, from a committee's vote to a contest of thousands of candidates.
``closure``   the strongest paths of a preference matrix that is already on the GPU, in each lane
              mode: 0 (chosen on the device), 16 and 32 bits.
``tally``     ballots on the GPU to the preference matrix: complete rankings, or ragged ballots
              that name only some of the candidates.
``rank``      wins and order of a strongest-path matrix.
``batch``     many elections of uneven size, prepared once and replayed as one CUDA graph.
``host``      the drop-in call: a NumPy matrix in, a NumPy matrix out.

Ballots come from a random-utility model: every candidate has a quality, every voter sees it
with noise and ranks by what it sees. ``spread`` is the qualities' range in units of the noise
(0 gives uniform permutations, the benchmark's other input).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from scalingelections_b200 import api
from scalingelections_b200.batch import BatchedElections, lanes_for_voters


# ------------------------------------------------------------------------------------------
# Cases
# ------------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # The reference script's default election (128 candidates, 2000 voters): the call where
        # latency, launches and host work count.
        {"name": "election-128", "kind": "election", "C": 128, "V": 2000, "spread": 2.0, "ragged": False},
        # A mid-size contest at an odd size with the default lanes.
        {"name": "closure-517-auto", "kind": "closure", "C": 517, "V": 1000, "spread": 2.0, "lanes": 0},
        # A national-scale candidate list, lanes known from the number of voters.
        {"name": "closure-1024-u16", "kind": "closure", "C": 1024, "V": 2000, "spread": 2.0, "lanes": 16},
        # The reference's random benchmark matrix with counts past 16 bits (V = 0: no ballots).
        {"name": "closure-1500-u32", "kind": "closure", "C": 1500, "V": 0, "spread": 0.0, "lanes": 32},
        # The largest election of the batched workload, closed alone.
        {"name": "closure-2048-auto", "kind": "closure", "C": 2048, "V": 4096, "spread": 2.0, "lanes": 0},
        # The single-election configuration: 4096 candidates, 4096 uniform ballots.
        {"name": "closure-4096-u16", "kind": "closure", "C": 4096, "V": 4096, "spread": 0.0, "lanes": 16},
        # The headline: 16384 candidates, 4096 correlated ballots.
        {"name": "closure-16384-u16", "kind": "closure", "C": 16384, "V": 4096, "spread": 2.0, "lanes": 16},
        # The single-election configuration's tally.
        {"name": "tally-4096", "kind": "tally", "C": 4096, "V": 4096, "spread": 0.0, "ragged": False},
        # Many voters who each rank a few or all of 1000 candidates.
        {"name": "tally-1000-ragged", "kind": "tally", "C": 1000, "V": 60000, "spread": 2.0, "ragged": True},
        # Winner and order of a large contest, at an odd size.
        {"name": "rank-10007", "kind": "rank", "C": 10007},
        # Mixed elections of a polling service, sizes log-uniform in [8, 2048].
        {"name": "batch-20", "kind": "batch", "n": 20, "c_max": 2048},
        # The reference script's own call, host memory to host memory.
        {"name": "host-4096", "kind": "host", "C": 4096, "V": 4096, "spread": 2.0},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["election", "election", "closure", "closure", "closure", "closure", "tally", "tally", "rank",
                       "batch", "host"])
    spread = rng.choice([0.0, 0.5, 2.0, 8.0])
    if kind == "election":
        return {"kind": kind, "C": _log_int(rng, 3, 2500), "V": _log_int(rng, 10, 20000), "spread": spread,
                "ragged": rng.random() < 0.3}
    if kind == "closure":
        lanes = rng.choice([0, 0, 16, 16, 32])
        C = _log_int(rng, 16, 5000 if lanes == 32 else 12000)
        V = 0 if lanes == 32 and rng.random() < 0.5 else _log_int(rng, 50, 8000)
        return {"kind": kind, "C": C, "V": V, "spread": spread, "lanes": lanes}
    if kind == "tally":
        C = _log_int(rng, 16, 6000)
        return {"kind": kind, "C": C, "V": _log_int(rng, 50, min(200000, 60000000 // C)), "spread": spread,
                "ragged": rng.random() < 0.5}
    if kind == "rank":
        return {"kind": kind, "C": _log_int(rng, 16, 16384)}
    if kind == "batch":
        return {"kind": kind, "n": rng.randint(4, 21), "c_max": _log_int(rng, 64, 2048)}
    return {"kind": kind, "C": _log_int(rng, 64, 6000), "V": _log_int(rng, 50, 8000), "spread": spread}


# ------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------
def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ballots(C: int, V: int, spread: float, g: torch.Generator) -> torch.Tensor:
    """V ballots over C candidates, int32 [V, C], most preferred first."""
    quality = torch.linspace(0.0, spread, C, device="cuda")[torch.randperm(C, generator=g, device="cuda")]
    out = torch.empty((V, C), dtype=torch.int32, device="cuda")
    step = max(1, (1 << 25) // C)
    for lo in range(0, V, step):
        hi = min(V, lo + step)
        noise = torch.randn((hi - lo, C), generator=g, device="cuda")
        out[lo:hi] = torch.argsort(noise - quality, dim=1).to(torch.int32)
    return out


def _csr(ballots: torch.Tensor, ragged: bool, g: torch.Generator) -> tuple[torch.Tensor, torch.Tensor]:
    """Ballots in CSR form; ragged ones keep their first 1 .. C names."""
    V, C = ballots.shape
    if not ragged:
        return ballots.reshape(-1), torch.arange(V + 1, dtype=torch.int64, device="cuda") * C
    lens = torch.randint(1, C + 1, (V,), generator=g, device="cuda")
    offsets = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=offsets[1:])
    keep = torch.arange(C, device="cuda")[None, :] < lens[:, None]
    return ballots[keep], offsets


def _matrix(C: int, V: int, spread: float, g: torch.Generator) -> torch.Tensor:
    """A preference matrix, uint32 [C, C]: the tally of V ballots, or random counts for V = 0."""
    if V == 0:
        return torch.randint(-(1 << 31), 1 << 31, (C, C), generator=g, device="cuda", dtype=torch.int32).view(torch.uint32)
    ids, offsets = _csr(_ballots(C, V, spread, g), False, g)
    return api.tally_device(ids, offsets, C)


def _batch_specs(case: dict, seed: int) -> list[tuple[int, int]]:
    """(C, V) of each election: sizes spread evenly over the logarithm of [8, c_max], so that
    another seed gives other elections of the same weight."""
    rng = random.Random(int(seed))
    n, c_max = case["n"], case["c_max"]
    return [(max(8, round(8 * (c_max / 8) ** (i / (n - 1)))), _log_int(rng, 50, 20000)) for i in range(n)]


def prepare(case: dict, seed: int):
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("election", "tally"):
        ids, offsets = _csr(_ballots(case["C"], case["V"], case["spread"], g), case["ragged"], g)
        return {"kind": kind, "C": case["C"], "ids": ids, "offsets": offsets}
    if kind == "closure":
        return {"kind": kind, "lanes": case["lanes"], "d": _matrix(case["C"], case["V"], case["spread"], g)}
    if kind == "rank":
        # Strengths of a contest decided by quality and noise, as a closure leaves them: any
        # matrix with a zero diagonal ranks at the same cost.
        C = case["C"]
        quality = torch.rand(C, generator=g, device="cuda")
        S = torch.rand((C, C), generator=g, device="cuda") + quality[:, None] - quality[None, :]
        S = (S.clamp_(min=0.0) * 2000.0).to(torch.int32)
        S.fill_diagonal_(0)
        return {"kind": kind, "S": S.view(torch.uint32)}
    if kind == "batch":
        specs = _batch_specs(case, seed)
        mats = [_matrix(C, V, 2.0, g) for C, V in specs]
        batch = BatchedElections(mats, [lanes_for_voters(V) for _, V in specs])
        batch.build_graph()
        return {"kind": kind, "batch": batch, "mats": mats}
    d = _matrix(case["C"], case["V"], case["spread"], g)
    return {"kind": kind, "P": d.view(torch.int32).cpu().numpy().view(np.uint32)}


# ------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "election":
        d = api.tally_device(state["ids"], state["offsets"], state["C"])
        S = api.strongest_paths_device(d)
        wins, ranking = api.rank_device(S)
        return {"d": d.view(torch.int32), "S": S.view(torch.int32), "wins": wins, "ranking": ranking}
    if kind == "closure":
        return api.strongest_paths_device(state["d"], lanes=state["lanes"]).view(torch.int32)
    if kind == "tally":
        return api.tally_device(state["ids"], state["offsets"], state["C"]).view(torch.int32)
    if kind == "rank":
        wins, ranking = api.rank_device(state["S"])
        return {"wins": wins, "ranking": ranking}
    if kind == "batch":
        b = state["batch"]
        b.launch_graph()
        return {"S": [s.view(torch.int32) for s in b.strongest_paths], "wins": b.wins, "rankings": b.rankings}
    return api.compute_strongest_paths(state["P"], allow_gpu=True, tile_size=32).view(np.int32)


# ------------------------------------------------------------------------------------------
# What a pass cannot do without, and what it has to return
# ------------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    """Bytes: every input read once, every output written once. Operations: two (a minimum and a
    maximum) per relaxation of the C^3 of a closure; one per pair of candidates and voter of a
    tally; one comparison per pair of candidates of a ranking."""
    kind = case["kind"]

    def closure(C):
        return {"bytes": 8.0 * C * C, "flops": 2.0 * C ** 3}

    def tally(C, V, ragged):
        return {"bytes": 4.0 * V * C * (0.5 if ragged else 1.0) + 8.0 * (V + 1) + 4.0 * C * C,
                "flops": 0.5 * V * C * C}

    def rank(C):
        return {"bytes": 4.0 * C * C + 8.0 * C, "flops": 0.5 * C * C}

    if kind in ("closure", "host"):
        return closure(case["C"])
    if kind == "tally":
        return tally(case["C"], case["V"], case["ragged"])
    if kind == "rank":
        return rank(case["C"])
    if kind == "election":
        C = case["C"]
        t = tally(C, case["V"], case["ragged"])
        return {"bytes": t["bytes"] + 4.0 * C * C + 8.0 * C, "flops": t["flops"] + 2.0 * C ** 3 + 0.5 * C * C}
    parts = [closure(C) for C, _ in _batch_specs(case, 0)]
    ranks = [rank(C) for C, _ in _batch_specs(case, 0)]
    return {"bytes": sum(p["bytes"] for p in parts) + sum(8.0 * C for C, _ in _batch_specs(case, 0)),
            "flops": sum(p["flops"] for p in parts + ranks)}


_EXACT_MAX_C = 5000  # a closure of int64 cells by single pivots takes seconds above this


def _exact_tally(ids: torch.Tensor, offsets: torch.Tensor, C: int) -> torch.Tensor:
    V = offsets.numel() - 1
    lens = offsets[1:] - offsets[:-1]
    voter = torch.repeat_interleave(torch.arange(V, device="cuda"), lens)
    place = torch.arange(ids.numel(), device="cuda") - offsets[:-1][voter]
    # Candidates a ballot does not name follow in ascending order.
    pos = torch.arange(C, device="cuda", dtype=torch.int32)[None, :] + C
    pos = pos.repeat(V, 1)
    pos[voter, ids.long()] = place.to(torch.int32)
    d = torch.empty((C, C), dtype=torch.int64, device="cuda")
    for i in range(C):
        d[i] = (pos[:, i:i + 1] < pos).sum(0)
    return d


def _exact_closure(d: torch.Tensor) -> torch.Tensor:
    S = torch.where(d > d.T, d, torch.zeros_like(d))
    S.fill_diagonal_(0)
    for k in range(S.shape[0]):
        S = torch.maximum(S, torch.minimum(S[:, k:k + 1], S[k:k + 1, :]))
    S.fill_diagonal_(0)
    return S


def _exact_rank(S: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    wins = (S > S.T).sum(1)
    return wins, torch.argsort(wins, descending=True, stable=True)


def _int64(t: torch.Tensor) -> torch.Tensor:
    return t.view(torch.int32).to(torch.int64) & 0xFFFFFFFF


def _int32(t: torch.Tensor) -> torch.Tensor:
    """Values of [0, 2^32) as the bit pattern that an int32 view of uint32 shows."""
    return torch.where(t >= 1 << 31, t - (1 << 32), t).to(torch.int32)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("election", "closure", "host") and case["C"] > _EXACT_MAX_C:
        return None
    state = prepare(case, seed)
    if kind == "election":
        d = _exact_tally(state["ids"], state["offsets"], case["C"])
        S = _exact_closure(d)
        wins, ranking = _exact_rank(S)
        return {"d": _int32(d), "S": _int32(S), "wins": wins.to(torch.int32), "ranking": ranking.to(torch.int32)}
    if kind == "closure":
        return _int32(_exact_closure(_int64(state["d"])))
    if kind == "tally":
        return _int32(_exact_tally(state["ids"], state["offsets"], case["C"]))
    if kind == "rank":
        wins, ranking = _exact_rank(_int64(state["S"]))
        return {"wins": wins.to(torch.int32), "ranking": ranking.to(torch.int32)}
    if kind == "batch":
        S = [_exact_closure(_int64(m)) for m in state["mats"]]
        ranked = [_exact_rank(s) for s in S]
        return {"S": [_int32(s) for s in S], "wins": [w.to(torch.int32) for w, _ in ranked],
                "rankings": [r.to(torch.int32) for _, r in ranked]}
    P = torch.from_numpy(state["P"].view(np.int32)).cuda()
    return _int32(_exact_closure(_int64(P.view(torch.uint32)))).cpu().numpy()
