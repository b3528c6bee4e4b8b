"""Which bounded solves try the class join: decided on the host from the bounds, before any launch."""
import contextlib
import math
import random

import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.bsolve import BoundedSolve, bounded_pools, bounded_share, caps
from carmichael_frontier_b200.workloads import draw_modulus, eligible_pool


def instance(seed, k, n, r, slack):
    while True:
        M = draw_modulus(seed)
        Q = eligible_pool(M, 10 ** 5)
        if len(Q) >= k + n:
            return Instance.build(M, Q[:k + n], Q[:k], r, int(math.prod(Q[:k]) * slack))
        seed += 1000


@pytest.mark.parametrize("seed,k,n,r,slack", [(1, 64, 100, 5, 10), (2, 64, 140, 4, 10), (3, 78, 159, 4, 10 ** 4),
                                              (4, 90, 60, 6, 10 ** 3), (5, 100, 200, 3, 30), (6, 76, 40, 6, 300)])
def test_share_estimate(seed, k, n, r, slack):
    x = instance(seed, k, n, r, slack)
    Icap, Dmin = caps(x)
    skip, INS = bounded_pools(x, Icap, Dmin)
    B0 = x.B0[skip:]
    rng = random.Random(seed)
    draws = 4000                                   # standard error of a share below 0.008
    share = lambda P, f: sum(f(math.prod(rng.sample(P, r))) for _ in range(draws)) / draws
    nD, nI = math.comb(len(B0), r), math.comb(len(INS), r)
    want = (share(B0, lambda p: p >= Dmin) * nD + share(INS, lambda p: p < Icap) * nI) / (nD + nI)
    got = bounded_share(B0, INS, r, Icap, Dmin)
    assert abs(got - want) < (0.06 if 0.05 <= got < 0.4 else 0.25)


@pytest.mark.parametrize("k,n,r,slack,tried", [(64, 100, 5, 10, False), (64, 140, 4, 10, False), (98, 163, 6, 10, False),
                                               (64, 60, 3, 10 ** 8, False), (78, 159, 4, 10 ** 4, True),
                                               (64, 70, 5, 10 ** 4, True)])
def test_hard_bounds_go_to_the_level_loop_at_once(monkeypatch, k, n, r, slack, tried):
    class Upload(Exception):
        pass

    def upload(self, parts):
        raise Upload

    monkeypatch.setattr(BoundedSolve, "_upload", upload)
    x = instance(7, k, n, r, slack)
    b = object.__new__(BoundedSolve)               # its generator needs a device; the route does not
    b.s = Solver("cuda", tuning=Tuning(strategy="bounded"))
    b.lib, b.torch = b.s.lib, b.s.torch
    monkeypatch.setattr(b.torch.cuda, "stream", lambda st: contextlib.nullcontext())
    monkeypatch.setattr(b.torch.cuda, "current_stream", lambda *a: None)
    if tried:
        with pytest.raises(Upload):
            b._join_class(x, *caps(x))
    else:
        assert b._join_class(x, *caps(x)) is None


def test_pools_of_a_bound_by_search_equal_the_definition():
    rng = random.Random(5)
    for seed in range(40):
        r = rng.choice((3, 4, 6, 8))
        x = instance(seed, rng.randint(r, 70), rng.randint(r, 90), r, 10 ** rng.uniform(-3, 9))
        for Icap, Dmin in (caps(x), (2, 1), (math.prod(x.INS[:r]), math.prod(x.B0[-r:])),
                           (x.INS[-1] * math.prod(x.INS[:r - 1]), x.B0[0] * math.prod(x.B0[-(r - 1):]) + 1)):
            small, large = math.prod(x.INS[:r - 1]), math.prod(x.B0[-(r - 1):])
            INS = [q for i, q in enumerate(x.INS) if i < r or q * small < Icap]
            skip = next((i for i in range(len(x.B0) - r) if x.B0[i] * large >= Dmin), len(x.B0) - r)
            assert bounded_pools(x, Icap, Dmin) == (skip, INS)
