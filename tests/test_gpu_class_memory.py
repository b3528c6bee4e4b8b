"""Device memory of the class join: solves that it does not leave room for take the other join."""
import math

import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.bsolve import BoundedSolve
from carmichael_frontier_b200.portfolio import BatchSolver, BatchTuning
from carmichael_frontier_b200.workloads import eligible_pool

pytestmark = pytest.mark.gpu
M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
Q = eligible_pool(M, 10 ** 5)


def instance(k, n, r, slack=10 ** 8):
    return Instance.build(M, Q[:k + n], Q[:k], r, math.prod(Q[:k]) * slack)


def summary(r):
    return (r.n_D, r.n_I, r.residue_pairs, r.screened, r.above_bound, r.rejected, r.pairs, [h.n for h in r.hits])


@pytest.fixture
def full(monkeypatch):
    """A device without room for a class workspace."""
    import torch
    real = Solver._buf

    def buf(self, name, nbytes):
        if name == "class":
            raise torch.OutOfMemoryError("no room")
        return real(self, name, nbytes)

    monkeypatch.setattr(Solver, "_buf", buf)


def test_solves_without_room_take_the_table_join(cuda, full):
    insts = [instance(64, n, 4) for n in (90, 110, 100)]
    tu = Tuning(class_min_probe=0)
    want = [summary(r) for r in Solver(cuda, tuning=Tuning(class_join=False)).solve_many(insts)]
    got = [Solver(cuda, tuning=tu).solve_instance(x) for x in insts]
    assert [summary(r) for r in got] == want and all(r.plan["no_class"] for r in got)
    marks = []
    assert summary(Solver(cuda, tuning=tu).solve_instance(insts[0], marks=marks)) == want[0]
    assert [t for t, _ in marks] == ["start", "gen_D", "probe", "check"]
    assert [summary(r) for r in Solver(cuda, tuning=tu).solve_many(insts)] == want
    b = BatchSolver(cuda, tuning=BatchTuning(dtab=tu))
    prep = b.prepare(insts)
    assert len(prep.single) == 3 and [summary(r) for r in b.run(prep)] == want


def test_bounded_solves_without_room_take_the_level_loop(cuda, full, monkeypatch):
    x = instance(64, 200, 4, 10 ** 4)
    ref = Solver(cuda, tuning=Tuning(strategy="bounded", class_join=False)).solve_instance(x)
    monkeypatch.setattr(BoundedSolve, "CLASS_MIN", 0)
    got = Solver(cuda, tuning=Tuning(strategy="bounded", class_min_probe=0)).solve_instance(x)
    assert summary(got) == summary(ref) and got.plan.get("table") != "class"


def test_a_growing_buffer_frees_the_old_one_first(cuda):
    import torch
    s = Solver(cuda)
    torch.cuda.empty_cache()
    base = torch.cuda.memory_allocated()
    s._buf("x", 2 << 30)
    torch.cuda.reset_peak_memory_stats()
    assert s._buf("x", (2 << 30) + 1).numel() == (2 << 30) + (64 << 20)
    assert torch.cuda.max_memory_allocated() - base <= (2 << 30) + (65 << 20)
