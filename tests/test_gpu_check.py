"""The warp-per-pair exact check at its edges: base sizes around a warp, size bounds at a hit."""
import math

import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.workloads import eligible_pool

M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13


@pytest.mark.gpu
@pytest.mark.parametrize("k", [2, 30, 31, 32, 33, 62, 64, 100])
def test_size_bound_and_korselt_against_integers(cuda, k):
    Q = eligible_pool(M, None)
    B0, INS, r = Q[:k], Q[k:k + 70], 2
    P0 = math.prod(B0)
    res = {}
    for i in range(len(INS)):
        for j in range(i):
            res.setdefault(P0 * INS[i] * INS[j] % M, []).append((INS[j], INS[i]))
    ns = sorted(P0 // (B0[x] * B0[y]) * p * q for x in range(k) for y in range(x) for p, q in res.get(B0[x] * B0[y] % M, []))
    if not ns:
        pytest.skip("no equal-residue pair")
    s = Solver(cuda, tuning=Tuning(strategy="fused"))
    for B in {ns[0], ns[0] - 1, ns[len(ns) // 2], ns[len(ns) // 2] - 1, ns[-1]}:
        if B < 1 or B.bit_length() > 2048:
            continue
        out = s.solve_instance(Instance.build(M, B0 + INS, B0, r, B))
        assert out.residue_pairs == len(ns) and out.rejected == 0
        assert [h.n for h in out.hits] == [n for n in ns if n <= B]
