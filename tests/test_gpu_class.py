"""The class join against the table join and the exhaustive product, over the forms it accepts."""
import math
import random

import numpy as np
import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200 import _lib
from carmichael_frontier_b200.workloads import eligible_pool

MODULI = {                                 # smooth even moduli
    "2^43": 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29,
    "2^46": 2 ** 7 * 3 ** 4 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 41,
    "2^51": 2 ** 7 * 3 ** 4 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29 * 37,
}


def summary(r):
    return (r.n_D, r.n_I, r.residue_pairs, r.screened, r.above_bound, r.rejected, r.pairs, [h.n for h in r.hits])


def instance(name, k, n_ins, r):
    M = MODULI[name]
    Q = eligible_pool(M, 10 ** 5)
    assert len(Q) >= k + n_ins, len(Q)
    Q = Q[:k + n_ins]
    return Instance.build(M, Q, Q[:k], r, math.prod(Q[:k]) * 10 ** 8)


@pytest.mark.gpu
@pytest.mark.parametrize("name,k,n_ins,r,window", [
    ("2^51", 64, 90, 2, None), ("2^43", 100, 440, 3, None), ("2^43", 64, 200, 4, None),
    ("2^43", 64, 197, 4, (1234, 40_000_001)),      # a window that starts and ends inside prefixes
    ("2^43", 50, 70, 5, None), ("2^46", 30, 63, 5, (777_777, 777_778)), ("2^51", 64, 150, 5, None),
    ("2^46", 64, 45, 5, None),                     # the I side builds
    ("2^43", 48, 53, 6, (3, 9_500_000)), ("2^43", 45, 44, 6, None), ("2^46", 40, 7, 6, None),
    ("2^43", 35, 36, 7, None), ("2^43", 32, 33, 8, None), ("2^43", 9, 9, 8, None),
])
def test_class_join_equals_table_join(cuda, name, k, n_ins, r, window):
    inst = instance(name, k, n_ins, r)
    lo, lim = window or (0, None)
    got = Solver(cuda, tuning=Tuning(class_min_probe=0)).solve_instance(inst, i_lo=lo, i_limit=lim)
    ref = Solver(cuda, tuning=Tuning(class_join=False)).solve_instance(inst, i_lo=lo, i_limit=lim)
    assert got.plan["class_plan"] and not ref.plan.get("class_plan")
    assert summary(got) == summary(ref)


@pytest.mark.gpu
def test_class_join_falls_back_when_a_survivor_list_runs_out(cuda, monkeypatch):
    inst = instance("2^46", 64, 97, 4)
    want = summary(Solver(cuda, tuning=Tuning(class_join=False)).solve_instance(inst))
    real = Solver._class_plan

    def short(self, x, plan):
        p = real(self, x, plan)
        if p is None:
            return None
        a = np.frombuffer(p, dtype=np.uint32).copy()
        a[18] = 1                                  # one chunk of survivors
        return a.tobytes()

    s = Solver(cuda, tuning=Tuning(class_min_probe=0))
    monkeypatch.setattr(Solver, "_class_plan", short)
    got = s.solve_instance(inst)
    assert got.plan["no_class"] and summary(got) == want


@pytest.mark.gpu
def test_class_join_in_a_list_of_solves(cuda):
    insts = [instance(n, 64, m, r) for n, m, r in (("2^46", 90, 4), ("2^51", 60, 5), ("2^46", 100, 4), ("2^51", 50, 5))]
    ref = [summary(x) for x in Solver(cuda, tuning=Tuning(class_join=False)).solve_many(insts)]
    s = Solver(cuda, tuning=Tuning(class_min_probe=0))
    for _ in range(2):
        assert [summary(x) for x in s.solve_many(insts)] == ref


def plan_of(m, nD, nI, r, i_lo=0, i_n=None, swap=0):
    lib = _lib.load()
    out = np.zeros(lib.cf_class_plan_bytes(), dtype=np.uint8)
    i_n = math.comb(nI, r) - i_lo if i_n is None else i_n
    assert lib.cf_class_plan(m, nD, nI, r, i_lo, i_n, swap, out.ctypes.data, out.nbytes) == _lib.CF_OK
    ok, d, mp, phi = out[8:24].view(np.uint32).tolist()
    return ok, d, mp, phi, out


def test_plan_takes_coprime_divisors_and_declines_the_rest():
    for M in MODULI.values():
        m = M // (M & -M)
        ok, d, mp, phi, _ = plan_of(m, 64, 100, 5)
        assert ok and m % d == 0 and m % mp == 0 and math.gcd(d, mp) == 1 and mp >= 1 << 27
        assert phi == sum(math.gcd(c, d) == 1 for c in range(d))
    assert not plan_of(3 ** 20, 64, 100, 3)[0]                 # too few classes
    assert not plan_of(3 ** 4 * 37 * 41 * 43, 64, 100, 3)[0]   # too small a modulus for the filter
    assert not plan_of((1 << 61) - 1, 64, 100, 5)[0]           # a large prime
    assert not plan_of(3 ** 39, 64, 100, 9)[0]                 # radius above 8
    assert not plan_of(MODULI["2^51"] >> 7, 64, 100, 5, i_n=0)[0]


def test_scaled_residues_of_equal_records_differ_by_at_most_one():
    rng = random.Random(1)
    for mp in ((1 << 27) + 1, 3 ** 20, 3968733375, (1 << 32) - 1):
        for _ in range(2000):
            x = rng.randrange(1, mp)
            vs = []
            for _ in range(2):                     # two factorisations of the same residue
                s = rng.randrange(1, mp)
                while math.gcd(s, mp) != 1:
                    s = rng.randrange(1, mp)
                q = x * pow(s, -1, mp) % mp
                w = (q << 64) // mp
                vs.append(((w >> 32) * s + ((w & 0xffffffff) * s >> 32)) & 0xffffffff)
            exact = (x << 32) // mp
            assert all(v in (exact, exact - 1) for v in vs), (mp, x, vs)


@pytest.mark.gpu
def test_portfolio_sends_moduli_to_the_class_join(cuda):
    from carmichael_frontier_b200.portfolio import BatchSolver, BatchTuning
    insts = [instance("2^46", 64, 100, 4), instance("2^51", 64, 40, 5), instance("2^43", 20, 30, 3), instance("2^46", 64, 90, 5)]
    lim = 1 << 20
    dt = Tuning(class_min_probe=1 << 18)
    bs = BatchSolver(cuda, tuning=BatchTuning(dtab=dt))
    prep = bs.prepare(insts, i_limit=lim)
    assert sorted(prep.single) == [0, 1, 3] and [b.idx for b in prep.batches] == [[2]]
    ref = [summary(x) for x in BatchSolver(cuda, tuning=BatchTuning(class_join=False)).solve(insts, i_limit=lim)]
    for graphs in (False, True, True):
        assert [summary(x) for x in bs.run(prep, graphs=graphs)] == ref
