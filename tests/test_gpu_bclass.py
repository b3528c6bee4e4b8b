"""Bounded solves through the class join, and the bounded side counts, against the level expansion."""
import math
import random

import numpy as np
import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning, _lib
from carmichael_frontier_b200.bsolve import BoundedSolve, caps
from carmichael_frontier_b200.tables import pool_table_host
from carmichael_frontier_b200.workloads import eligible_pool

M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
Q = eligible_pool(M, 10 ** 5)


def summary(r):
    return (r.n_D, r.n_I, r.residue_pairs, r.screened, r.above_bound, r.rejected, r.pairs, [h.n for h in r.hits])


def counts(cuda, B0, INS, r, Icap, Dmin):
    import torch
    b = BoundedSolve(Solver(cuda))
    lib = _lib.load()
    out = torch.zeros(2, dtype=torch.int64, device=cuda)
    up = lambda a: torch.from_numpy(a.view(np.uint8).copy()).to(cuda)
    tabs = [up(pool_table_host(B0, r, M, 1)), up(b._bound_table(lib.cf_ddump_bounds, B0, r, Dmin)),
            up(pool_table_host(INS, r, M, 1)), up(b._bound_table(lib.cf_igen_bounds, INS, r, Icap))]
    p = [t.data_ptr() for t in tabs]
    _lib.check(lib.cf_bounded_count(1, p[0], p[1], len(B0), r, out.data_ptr(), None), "D")
    _lib.check(lib.cf_bounded_count(0, p[2], p[3], len(INS), r, out.data_ptr() + 8, None), "I")
    torch.cuda.synchronize()
    return out.tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("r", [3, 4, 5, 6, 8])
def test_counts_equal_brute_force(cuda, r):
    from itertools import combinations
    rng = random.Random(r)
    nb, ni = r + 4, r + 6
    B0, INS = Q[:nb], Q[nb:nb + ni]
    pD = sorted(math.prod(c) for c in combinations(B0, r))
    pI = sorted(math.prod(c) for c in combinations(INS, r))
    for _ in range(4):
        d, i = rng.choice(pD), rng.choice(pI)
        for dd, ii in ((d, i), (d + 1, i + 1), (0, pI[-1] + 1), (pD[-1] + 1, 2)):
            assert counts(cuda, B0, INS, r, ii, dd) == [sum(x >= dd for x in pD), sum(x < ii for x in pI)]


@pytest.mark.gpu
@pytest.mark.parametrize("k,n,r,slack", [(64, 200, 4, 10 ** 4), (64, 200, 4, 7), (80, 110, 4, 10 ** 12), (40, 60, 5, 10 ** 3),
                                         (30, 52, 5, 20), (36, 40, 6, 10 ** 2), (26, 30, 7, 10 ** 6), (24, 26, 8, 10 ** 10)])
def test_bounded_solve_equals_level_expansion(cuda, k, n, r, slack, monkeypatch):
    B0 = Q[:k]
    inst = Instance.build(M, Q[:k + n], B0, r, math.prod(B0) * slack)
    ref = Solver(cuda, tuning=Tuning(strategy="bounded", class_join=False)).solve_instance(inst)
    monkeypatch.setattr(BoundedSolve, "CLASS_MIN", 0)
    monkeypatch.setattr(BoundedSolve, "CLASS_RATIO", 1 << 60)
    got = Solver(cuda, tuning=Tuning(strategy="bounded", class_min_probe=0)).solve_instance(inst)
    assert summary(got) == summary(ref)
    assert got.plan["table"] == "class" and ref.plan.get("table") != "class"


@pytest.mark.gpu
def test_bounds_at_a_pair(cuda, monkeypatch):
    """Dmin and Icap exactly at a pair's products keep it or drop it as the level expansion does."""
    B0 = Q[:64]
    inst = Instance.build(M, Q[:264], B0, 4, math.prod(B0) * 10 ** 4)
    monkeypatch.setattr(BoundedSolve, "CLASS_MIN", 0)
    monkeypatch.setattr(BoundedSolve, "CLASS_RATIO", 1 << 60)
    s = Solver(cuda, tuning=Tuning(strategy="bounded", class_min_probe=0))
    t = Solver(cuda, tuning=Tuning(strategy="bounded", class_join=False))
    b, lev = BoundedSolve(s), BoundedSolve(t)
    Icap, _ = caps(inst)
    pairs, _, _, _ = lev._join(inst, Icap, 0, None, None)
    assert pairs
    for dd, ii in pairs[:3]:
        D, I = math.prod(inst.B0[x] for x in dd), math.prod(inst.INS[x] for x in ii)
        for Ic, Dm in ((I + 1, D), (I, D), (I + 1, D + 1)):
            got = b._join_class(inst, Ic, Dm)
            ref = lev._join(inst, Ic, Dm, None, None)
            assert got is not None and sorted(got[0]) == sorted(ref[0]) and got[1:3] == ref[1:3]


@pytest.mark.gpu
def test_counts_by_walking_equal_the_level_expansion(cuda):
    """C(n, r-2) above 2^20 prefixes: the walking form of the count kernel."""
    B0, INS, r = Q[:76], Q[76:176], 6
    assert math.comb(76, r - 2) > 1 << 20
    g = BoundedSolve(Solver(cuda)).gen
    Dmin = math.prod(B0[-6:]) * 2 // 3
    Icap = math.prod(INS[:6]) * 3
    nD = g.generate_D(B0, r, M, Dmin, bitmask=2)[2]
    it = g.generate_I(INS, r, M, 1, Icap)
    nI = sum(k.numel() for k, _ in it)
    assert nD and nI and counts(cuda, B0, INS, r, Icap, Dmin) == [nD, nI]
