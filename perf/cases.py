"""Workloads of the residue join, as a program that uses the package runs them.

Each case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` one more
from the same ranges; ``prepare`` makes what a program holds before the call (moduli, pools and
bounds as Python integers for the solvers, key and id tensors on the GPU for the record
functions), ``run`` is one pass through the public entry points, ``work`` the bytes and operations
a pass cannot do without, and ``exact`` the result in plain Python or numpy where that is quick.

Kinds of case:

  solve      ``solve`` on one modulus: every pair of an r-subset of the k smallest pool primes
             and an r-subset of the rest with equal residues, checked against the size bound
  campaign   ``solve_many`` on a list of moduli, the way a search goes through its moduli
  portfolio  ``BatchSolver.solve`` on moduli of uneven pools and radii 4, 5, 6, a bounded window
             of the I side each
  bounded    ``solve(strategy="auto")`` with a tight size bound, the request of a serving loop
  sort       ``mitm_gpu2.sort_side`` of one materialised side
  dropin     ``generate``, ``sort_side``, ``join_sorted`` on both sides of one modulus, the
             reference module's own call sequence
  igen       ``igen_gpu.generate``: the records of a product-bounded side
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import carmichael_frontier_b200 as cf
from carmichael_frontier_b200 import igen_gpu, mitm_gpu2
from carmichael_frontier_b200.portfolio import BatchSolver
from carmichael_frontier_b200.workloads import draw_modulus, eligible_pool

DEVICE = "cuda"
PRIME_CAP = 10 ** 5          # pools hold primes below this
MAX_RECORDS = 1.0e9          # drawn joins: records of both sides
MAX_SORT = 1 << 26


def listed():
    return [
        # the smallest call: the k = 29, r = 2 instance, a few thousand records, all launches and host work
        {"name": "solve_k29_r2", "kind": "solve", "k": 29, "pool": 120, "r": 2, "small_modulus": True},
        # one modulus of the k = 64 search at the radius most of its time goes to, |INS| = 150
        {"name": "solve_k64_r5", "kind": "solve", "k": 64, "pool": 214, "r": 5, "small_modulus": False},
        # a search over moduli one after another (radius 5, smaller pools): host and device work overlap
        {"name": "campaign_k64_r5", "kind": "campaign", "k": 64, "pool": 190, "r": 5, "count": 6},
        # the large-radius instance: pool 160, r = 7, 6.2e8 D records against 1.2e10 I records
        {"name": "large_k64_r7", "kind": "solve", "k": 64, "pool": 160, "r": 7, "small_modulus": False},
        # a portfolio of uneven pools and mixed radii, I ranks [0, 2^24) of each
        {"name": "portfolio_r456", "kind": "portfolio", "k": 64, "pool_lo": 120, "pool_hi": 350, "count": 24,
         "i_limit": 1 << 24},
        # an ordinary serving request: a bound close to the base product, a few milliseconds
        {"name": "request_k78_r4", "kind": "bounded", "k": 78, "pool": 237, "r": 4},
        # a large serving request: radius 6 over a wide pool
        {"name": "request_k76_r6", "kind": "bounded", "k": 76, "pool": 200, "r": 6},
        # sides to sort: a small one of odd length, the k = 64, r = 5 D side, a large I chunk
        {"name": "sort_20k", "kind": "sort", "n": 20_003, "m_bits": 53, "dup": 0},
        {"name": "sort_7p6M", "kind": "sort", "n": math.comb(64, 5), "m_bits": 53, "dup": 0},
        {"name": "sort_64M", "kind": "sort", "n": 1 << 26, "m_bits": 61, "dup": 16},
        # the reference module's own sequence on one modulus at radius 4
        {"name": "dropin_k64_r4", "kind": "dropin", "k": 64, "pool": 190, "r": 4, "i_limit": 1 << 24},
        # the bounded producer on its own: 8e6 of 1.1e7 records lie under the product cap
        {"name": "igen_r4_8M", "kind": "igen", "k": 64, "pool": 194, "r": 4, "records": 8_000_000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "campaign", "portfolio", "bounded", "sort", "sort", "dropin",
                       "igen"))
    if kind == "solve":
        while True:
            r, k = rng.choice((2, 3, 4, 5, 5, 6)), rng.randint(24, 100)
            pool = rng.randint(k + 12, 320)
            n = math.comb(k, r) + math.comb(pool - k, r)
            if n <= MAX_RECORDS:
                return {"kind": "solve", "k": k, "pool": pool, "r": r, "small_modulus": False}
    if kind == "campaign":
        return {"kind": "campaign", "k": 64, "pool": rng.randint(130, 190), "r": rng.choice((4, 5)),
                "count": rng.randint(2, 6)}
    if kind == "portfolio":
        lo = rng.randint(100, 200)
        return {"kind": "portfolio", "k": 64, "pool_lo": lo, "pool_hi": lo + rng.randint(0, 150),
                "count": rng.randint(2, 16), "i_limit": _log_uniform(rng, 1 << 18, 1 << 24)}
    if kind == "bounded":
        r, k = rng.choice((3, 4, 5)), rng.randint(64, 100)
        return {"kind": "bounded", "k": k, "pool": rng.randint(k + 12, 300), "r": r}
    if kind == "sort":
        return {"kind": "sort", "n": _log_uniform(rng, 1000, MAX_SORT), "m_bits": rng.randint(50, 62),
                "dup": rng.choice((0, 0, 16, 1000))}
    if kind == "dropin":
        return {"kind": "dropin", "k": rng.randint(30, 64), "pool": rng.randint(80, 190), "r": rng.choice((3, 4)),
                "i_limit": _log_uniform(rng, 1 << 18, 1 << 24)}
    pool, r = rng.randint(130, 200), rng.choice((3, 4, 4))
    n = math.comb(pool - 64, r)
    return {"kind": "igen", "k": 64, "pool": pool, "r": r, "records": _log_uniform(rng, n // 100, n - 1)}


# -- inputs -----------------------------------------------------------------------

def _modulus(seed, pool, small=False):
    """(M, its `pool` smallest eligible primes): the first modulus after `seed` whose pool is large enough."""
    rng = random.Random(seed)
    while True:
        if small:            # around 2 * 10^7, as the k = 29 instance's modulus 21621600
            M = 2 ** rng.randint(4, 7) * 3 ** rng.randint(2, 4) * 5 ** rng.randint(1, 2) * 7 * 11 * 13
            M *= rng.choice((1, 17, 19))
        else:
            M = draw_modulus(rng.getrandbits(40))
        Q = eligible_pool(M, None if small else PRIME_CAP)
        if len(Q) >= pool:
            return M, Q[:pool]


def _instance(seed, c):
    M, Q = _modulus(seed, c["pool"], c.get("small_modulus", False))
    B0 = Q[:c["k"]]
    P0 = math.prod(B0)
    if c["kind"] == "bounded":
        B = P0 * 10 ** 4
    else:
        B = 10 ** 148 if c["k"] == 64 else P0 * 10 ** 8
    return M, Q, B0, c["r"], B


def _sub_seed(seed, i):
    return seed * 1009 + i


def _portfolio_shape(c, i):
    """Pool size and radius of a portfolio's i-th modulus."""
    span = c["pool_hi"] - c["pool_lo"]
    return c["pool_lo"] + span * ((i * 7) % c["count"]) // max(1, c["count"] - 1), (4, 5, 6)[i % 3]


def _side(c, seed, device):
    """Unsorted residue keys and packed ids of one side; `dup` of the records repeat earlier keys."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    hi = 3 << (c["m_bits"] - 2)
    keys = torch.randint(0, hi, (c["n"],), generator=g, device=device, dtype=torch.int64)
    ids = torch.randint(0, 1 << 50, (c["n"],), generator=g, device=device, dtype=torch.int64)
    if c["dup"]:
        d = min(c["dup"], c["n"] // 2)
        keys[-d:] = keys[:d]
    return keys.view(torch.uint64), ids.view(torch.uint64)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "bounded"):
        return {"case": case, "args": _instance(seed, case)}
    if kind == "campaign":
        return {"case": case, "insts": [_instance(_sub_seed(seed, i), case) for i in range(case["count"])]}
    if kind == "portfolio":
        insts = []
        for i in range(case["count"]):
            pool, r = _portfolio_shape(case, i)
            M, Q, B0, r, B = _instance(_sub_seed(seed, i), dict(case, pool=pool, r=r))
            insts.append(cf.Instance.build(M, Q, B0, r, B))
        return {"case": case, "insts": insts, "solver": BatchSolver(DEVICE)}
    if kind == "sort":
        keys, ids = _side(case, seed, DEVICE)
        return {"case": case, "keys": keys, "ids": ids}
    M, Q, B0, r, B = _instance(seed, case)
    INS = Q[case["k"]:]
    if kind == "dropin":
        return {"case": case, "M": M, "B0": B0, "INS": INS, "r": r, "P0": math.prod(B0)}
    return {"case": case, "M": M, "INS": INS, "r": r, "P0": math.prod(B0),
            "Icap": _cap_below(INS, r, case["records"])}


def _cap_below(primes, r, records):
    """The product with exactly `records` smaller ones among the products of r of the primes (r = 3, 4)."""
    lg = torch.tensor([math.log2(p) for p in primes], dtype=torch.float64, device=DEVICE)
    a = torch.triu_indices(len(primes), len(primes), 1, device=DEVICE)
    b = a if r == 4 else torch.arange(len(primes), device=DEVICE)[None, :]
    rows = (a[1][:, None] < b[0][None, :]).nonzero()
    first, last = a[:, rows[:, 0]], b[:, rows[:, 1]]
    lgs = lg[first].sum(0) + lg[last].sum(0)
    at = int(lgs.argsort()[records])
    return math.prod(primes[int(i)] for i in (*first[:, at], *last[:, at]))


# -- one pass ---------------------------------------------------------------------

def _rows(r):
    """Rows of a pair table: more than any instance of the ranges has pairs."""
    return {5: 1 << 12, 6: 1 << 14, 7: 1 << 16}.get(r, 1 << 8)


def _table(rows, n, width):
    out = np.full((max(n, len(rows)), width), -1, dtype=np.int64)
    if rows:
        out[:len(rows), :len(rows[0])] = np.array(rows, dtype=np.int64)
    return out


def _results(Ms, results, r, k, n):
    """The record a search keeps of each modulus: modulus and counts, every equal-residue pair
    (deleted and inserted primes; n rows), every hit's factors (n / 8 rows); tables padded with -1."""
    counts = [[M, x.n_D, x.n_I, x.residue_pairs, x.screened, x.above_bound, x.rejected]
              for M, x in zip(Ms, results)]
    return {"counts": np.array(counts, dtype=np.int64),
            "pairs": np.stack([_table([d + i for d, i in x.pairs], n, 2 * r) for x in results]),
            "hits": np.stack([_table([h.factors for h in x.hits], n // 8, k) for x in results])}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("solve", "bounded"):
        M, Q, B0, r, B = state["args"]
        res = cf.solve(M, Q, B0, r, B, strategy="auto" if kind == "bounded" else "fused")
        return _results([M], [res], r, case["k"], _rows(r))
    if kind == "campaign":
        return _results([x[0] for x in state["insts"]], cf.solve_many(state["insts"]), case["r"], case["k"],
                        _rows(case["r"]))
    if kind == "portfolio":
        solver = state["solver"]
        prep = solver.prepare(state["insts"], i_limit=case["i_limit"])
        out = solver.run(prep)
        solver.release(prep)
        return _results([x.M for x in state["insts"]], out, 6, case["k"], 256)
    if kind == "sort":
        keys, ids = mitm_gpu2.sort_side(state["keys"], state["ids"])
        return keys.view(torch.int64), ids.view(torch.int64)
    if kind == "dropin":
        M, r = state["M"], state["r"]
        bits = max(6, (max(len(state["B0"]), len(state["INS"])) - 1).bit_length())
        Dk, Did = mitm_gpu2.sort_side(*mitm_gpu2.generate(state["B0"], r, M, 1, bits))
        hi = min(case["i_limit"], math.comb(len(state["INS"]), r))
        Ik, Iid = mitm_gpu2.sort_side(*mitm_gpu2.generate(state["INS"], r, M, state["P0"] % M, bits, 0, hi))
        d, i = mitm_gpu2.join_sorted(Dk, Did, Ik, Iid)
        pairs = [x + y for x, y in zip(mitm_gpu2.decode_ids(d, r, bits), mitm_gpu2.decode_ids(i, r, bits))]
        return [x.view(torch.int64) for x in (Dk, Did, Ik, Iid)] + [_table(pairs, 256, 2 * r)]
    keys, ids, n = igen_gpu.generate(state["INS"], state["r"], state["M"], state["P0"], state["Icap"])
    return keys.view(torch.int64), ids.view(torch.int64), n


# -- what a pass cannot do without ------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 32 * case["n"], "flops": 0}                    # keys and ids read and written once
    if kind == "igen":
        return {"bytes": 16 * case["records"], "flops": case["records"]}   # one product a record, 16 bytes written
    if kind == "dropin":
        nD = math.comb(case["k"], case["r"])
        nI = min(case["i_limit"], math.comb(case["pool"] - case["k"], case["r"]))
        return {"bytes": 16 * (nD + nI), "flops": nD + nI}              # both sorted sides are results
    # the joins read a pool of primes and return a few pairs; the work is one modular product per record
    if kind == "portfolio":
        n = b = 0
        for i in range(case["count"]):
            pool, r = _portfolio_shape(case, i)
            n += math.comb(case["k"], r) + min(case["i_limit"], math.comb(pool - case["k"], r))
            b += 8 * pool
        return {"bytes": b, "flops": n}
    if kind == "bounded":
        return {"bytes": 8 * case["pool"], "flops": math.comb(case["k"], case["r"])}   # the D side (I depends on the bound)
    n = math.comb(case["k"], case["r"]) + math.comb(case["pool"] - case["k"], case["r"])
    m = case.get("count", 1)
    return {"bytes": 8 * case["pool"] * m, "flops": n * m}


def exact(case, seed):
    """The result in plain numpy, for the kinds where that is quick (every output is whole numbers)."""
    if case["kind"] != "sort" or case["n"] > 1 << 24:
        return None
    keys, ids = _side(case, seed, DEVICE if torch.cuda.is_available() else "cpu")
    k, i = keys.view(torch.int64).cpu().numpy(), ids.view(torch.int64).cpu().numpy()
    order = np.argsort(k, kind="stable")                                 # keys are below 2^63
    return k[order], i[order]
