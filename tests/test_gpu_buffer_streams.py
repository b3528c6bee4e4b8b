"""Solver buffers and streams: memory that a solver gives up is not handed out while its streams use it."""
import math

import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.workloads import eligible_pool

pytestmark = pytest.mark.gpu


def busy(torch, stream):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(600_000_000)             # a third of a second
        ev = torch.cuda.Event()
        ev.record(stream)
    return ev


def test_a_solver_of_its_own_stream(cuda):
    import torch
    st = torch.cuda.Stream(cuda)
    s = Solver(cuda, stream=st)
    n = 96 << 20
    old = s._buf("x", n).data_ptr()
    ev = busy(torch, st)
    s._buf("x", 2 * n)                             # the old block is freed while its stream is busy
    got = [torch.empty(n, dtype=torch.uint8, device=cuda) for _ in range(3)]
    assert not ev.query() and old not in [t.data_ptr() for t in got]
    torch.cuda.synchronize()


def test_a_solver_used_from_two_streams(cuda):
    import torch
    M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
    Q = eligible_pool(M, 10 ** 5)[:154]
    x = Instance.build(M, Q, Q[:64], 3, math.prod(Q[:64]) * 10 ** 8)
    s = Solver(cuda, tuning=Tuning(pair_capacity=1 << 16))          # result rows of 5.8 MB: a block of their own
    s.solve_instance(x)                            # buffers made on the default stream
    st = torch.cuda.Stream(cuda)
    with torch.cuda.stream(st):
        ev = busy(torch, st)
        s.enqueue(x, s._direct_plan(x, None))      # used on another one
    held = {t.data_ptr(): t.numel() for t in s._bufs.values() if t.numel() >= 2 << 20}   # blocks of their own
    assert held
    del s
    got = [torch.empty(n, dtype=torch.uint8, device=cuda) for n in held.values() for _ in range(2)]
    assert not ev.query() and not held.keys() & {t.data_ptr() for t in got}
    torch.cuda.synchronize()
