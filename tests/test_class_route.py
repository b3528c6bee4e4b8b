"""Which instances take the class join: decided on the host, so tested without a GPU."""
import math

import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.workloads import eligible_pool

M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
Q = eligible_pool(M, 10 ** 5)


def instance(k, n, r):
    return Instance.build(M, Q[:k + n], Q[:k], r, math.prod(Q[:k]) * 10 ** 8)


def class_plan(x, **tuning):
    s = Solver("cuda", tuning=Tuning(**tuning))
    nD, nI = math.comb(len(x.B0), x.r), math.comb(len(x.INS), x.r)
    return s._class_plan(x, s.plan(nD, nI))


@pytest.mark.parametrize("side", ["B0", "INS"])
def test_primes_of_2_31_or_more_do_not_take_the_class_join(side):
    # its kernels multiply 32-bit factors; Instance.build refuses such primes, the class itself does not
    x = instance(64, 120, 4)
    assert class_plan(x) is not None
    getattr(x, side)[-1] = (1 << 31) + 11
    x.P0 = math.prod(x.B0)
    assert class_plan(x) is None
