"""Parts of the class join that only large sides reach, and each of its lists run out, against the table join."""
import importlib
import math
import struct

import numpy as np
import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.workloads import draw_modulus, eligible_pool

pytestmark = pytest.mark.gpu
S = importlib.import_module("carmichael_frontier_b200.solve")     # the package's `solve` is the function


def summary(r):
    return (r.n_D, r.n_I, r.residue_pairs, r.screened, r.above_bound, r.rejected, r.pairs, [h.n for h in r.hits])


def instance(seed, k, n, r):
    while True:
        M = draw_modulus(seed)
        Q = eligible_pool(M, 10 ** 5)
        if len(Q) >= k + n:
            return Instance.build(M, Q[:k + n], Q[:k], r, math.prod(Q[:k]) * 10 ** 8)
        seed += 1


def table(cuda, x):
    return Solver(cuda, tuning=Tuning(class_join=False)).solve_instance(x)


def shape(cp):
    """(classes, list elements per thread, entries of the probing side's suffix blocks, their number)"""
    phi, = struct.unpack_from("<I", cp, 20)
    run, = struct.unpack_from("<I", cp, 44)
    side = struct.unpack_from("<15I", cp, 208 + 112)
    return phi, run, 32 * side[5], side[14] // (32 * side[5])


@pytest.mark.parametrize("seed,k,n,r,what", [
    (3, 64, 60, 6, "several classes per CTA"),           # 750 classes: build and resolve take five each
    (3, 50, 90, 7, "rounds"),                            # 1.0e8 against 7.5e9: list runs of 4, several resolve rounds,
])                                                       # long block ranges
def test_large_sides(cuda, seed, k, n, r, what):
    x = instance(seed, k, n, r)
    got = Solver(cuda).solve_instance(x)
    cp = got.plan["class_plan"]
    phi, run, block, blocks = shape(cp)
    assert phi > 148
    if what == "rounds":
        per = math.comb(k, r) / phi / 49152
        assert run == 4 and blocks >= 1 << 14
        assert math.comb(n, r) / phi * (per + per * per) / 256 > 2 * 65536     # survivors of a class
    assert summary(got) == summary(table(cuda, x))


@pytest.mark.parametrize("word,value", [(18, 1), (19, 1), (20, 16)])     # survivor chunks, candidates, kept records
def test_each_list_that_runs_out_sends_the_solve_to_the_table(cuda, monkeypatch, word, value):
    x = instance(5, 64, 90, 5)
    real = Solver._class_plan

    def short(self, inst, plan):
        p = real(self, inst, plan)
        if p is None:
            return None
        a = np.frombuffer(p, dtype=np.uint32).copy()
        assert a[word] > 1000
        a[word] = value
        return a.tobytes()

    want = summary(table(cuda, x))
    monkeypatch.setattr(Solver, "_class_plan", short)
    got = Solver(cuda).solve_instance(x)
    assert got.plan["no_class"] and summary(got) == want


def test_the_least_filter_modulus(cuda):
    # just above 2^27: one record pair in 2^27 agrees by chance, some 3,000 of a full round (8,192 fit)
    p = (1 << 27) + 29
    M = 2 ** 4 * 163 * p
    primes = [q for q in range(200, 3000) if all(q % d for d in range(2, int(q ** 0.5) + 1))][:64 + 180]
    x = Instance.build(M, primes, primes[:64], 5, math.prod(primes[:64]) * 10 ** 8)
    s = Solver(cuda)
    _ok, d, mp, phi, _ws = S.plan_head(s._direct_plan(x, None)["class_plan"])
    assert (d, mp, phi) == (163, p, 162)
    got = s.solve_instance(x, verify=False)
    assert got.plan["class_plan"] and got.residue_pairs > 10_000
    want = Solver(cuda, tuning=Tuning(class_join=False)).solve_instance(x, verify=False)
    assert summary(got) == summary(want)


def test_a_pair_buffer_that_runs_out_grows(cuda, monkeypatch):
    M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
    Q = eligible_pool(M, 10 ** 5)[:164]
    x = Instance.build(M, Q, Q[:64], 5, math.prod(Q[:64]) * 10 ** 8)
    want = table(cuda, x)
    assert want.residue_pairs > 16
    monkeypatch.setattr(S, "class_pairs", lambda *a: 4)
    got = Solver(cuda).solve_instance(x)
    assert got.plan["class_plan"] and got.plan["pairs"] > 4 and summary(got) == summary(want)
