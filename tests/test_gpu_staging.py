"""Page-locked staging of a solve: not rewritten while a queued solve may read it, freed memory kept
until the copies that use it have run."""
import math

import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.workloads import eligible_pool

pytestmark = pytest.mark.gpu
M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
Q = eligible_pool(M, 10 ** 5)
TUNINGS = [Tuning(), Tuning(class_min_probe=0), Tuning(class_join=False, part_min_buckets=16)]


def instance(k, n, r=3):
    return Instance.build(M, Q[:k + n], Q[:k], r, math.prod(Q[:k]) * 10 ** 8)


def summary(r):
    return (r.n_D, r.n_I, r.residue_pairs, r.screened, r.above_bound, r.rejected, r.pairs, [h.n for h in r.hits])


def busy(torch, stream):
    """Hold the stream for a third of a second; an event after it."""
    with torch.cuda.stream(stream):
        torch.cuda._sleep(600_000_000)
        ev = torch.cuda.Event()
        ev.record(stream)
    return ev


@pytest.mark.parametrize("tu", TUNINGS)
def test_a_second_solve_queued_before_the_first_is_collected(cuda, tu):
    import torch
    a, b = instance(64, 90), instance(60, 97)
    s = Solver(cuda, tuning=tu)
    want = [summary(s.solve_instance(x)) for x in (a, b)]
    st = torch.cuda.current_stream(cuda)
    for x, y, w in ((a, b, want), (b, a, want[::-1]), (a, a, [want[0]] * 2)):
        ev = busy(torch, st)
        h = s.enqueue(x, s._direct_plan(x, None))
        g = s.enqueue(y, s._direct_plan(y, None))
        assert not ev.query()                      # both are queued, no upload has run
        if "hread" in h:
            assert h["hread"].data_ptr() != g["hread"].data_ptr()
            assert summary(s.collect(x, h)[0]) == w[0]
        assert summary(s.collect(y, g)[0]) == w[1] and not s._queued


def test_freed_staging_waits_for_its_stream(cuda):
    import torch
    a = instance(64, 90)
    s = Solver(cuda)
    s.solve_instance(a)
    ev = busy(torch, torch.cuda.current_stream(cuda))
    s.enqueue(a, s._direct_plan(a, None))
    held = {t.data_ptr(): t.numel() for t, _ in s._pinned.values()}
    del s
    got = [torch.empty(n, dtype=torch.uint8, pin_memory=True) for n in held.values() for _ in range(2)]
    assert not ev.query() and not held.keys() & {t.data_ptr() for t in got}
    torch.cuda.synchronize()
