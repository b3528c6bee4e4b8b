"""The table join of sides that the class join would take: built in place and by ranges, one solve at a
time, in a list and in batches.  It remains the path of moduli without a class plan and after an overflow."""
import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.portfolio import BatchSolver, BatchTuning

pytestmark = pytest.mark.gpu


def as_lists(pairs):
    return sorted([list(D), list(I)] for D, I in pairs)


def summary(r):
    return (r.n_D, r.n_I, r.residue_pairs, r.screened, r.above_bound, r.rejected, sorted(r.pairs), [h.n for h in r.hits])


def instances(golden, count):
    return [Instance.build(g["M"], g["Q"], g["B0"], g["r"], int(g["B"])) for g in golden["config2"][:count]]


FORMS = {
    "in place": dict(part_build=False),
    "ranges": dict(part_min_buckets=16),
    "9-bit ranges": dict(part_min_buckets=16, part_lb=9),
    "ranges too small": dict(part_min_buckets=16, part_sigma=-6.0),
    "fuller buckets": dict(part_min_buckets=16, dtab_load=12.0),
}


@pytest.mark.parametrize("form", FORMS)
def test_table_builds_equal_the_class_join(cuda, golden, form):
    lim = 1 << 21
    s = Solver(cuda, tuning=Tuning(class_join=False, **FORMS[form]))
    for x in instances(golden, 2):
        want = Solver(cuda).solve_instance(x, i_limit=lim)
        assert want.plan["class_plan"]
        plan = s._direct_plan(x, lim)
        assert not plan["class_plan"] and (s._part_shape(x, plan) is None) == (form == "in place")
        got = s.solve_instance(x, i_limit=lim)
        assert summary(got) == summary(want) and not got.plan["class_plan"]
        assert bool(got.plan.get("no_part")) == (form == "ranges too small")


def test_whole_moduli_by_table_equal_the_reference(cuda, golden):
    s = Solver(cuda, tuning=Tuning(class_join=False))
    for g, x in zip(golden["config2"], instances(golden, 5)):
        got = s.solve_instance(x)
        assert not got.plan["class_plan"] and got.residue_pairs == g["matches"] and as_lists(got.pairs) == g["pairs"]


def test_partitioned_builds_in_a_list(cuda, golden):
    xs = instances(golden, 3)
    xs = xs + xs[::-1]
    lim = 1 << 22
    want = [summary(Solver(cuda).solve_instance(x, i_limit=lim)) for x in xs]
    s = Solver(cuda, tuning=Tuning(class_join=False, part_min_buckets=16))
    out = s.solve_many(xs, i_limit=lim)
    assert [summary(r) for r in out] == want
    assert all(not r.plan["class_plan"] and not r.plan.get("no_part") for r in out)
    half = s.solve_many(xs, i_limit=lim, i_lo=1 << 21)
    low = s.solve_many(xs, i_limit=1 << 21)
    for h, l, w in zip(half, low, want):
        assert h.n_I + l.n_I == w[1] and sorted(h.pairs + l.pairs) == w[6]


def test_batches_of_full_moduli_equal_the_reference(cuda, golden):
    b = BatchSolver(cuda, tuning=BatchTuning(class_join=False))
    prep = b.prepare(instances(golden, 5))
    assert not prep.single and sorted(k for x in prep.batches for k in x.idx) == list(range(5))
    for g, got in zip(golden["config2"], b.run(prep)):
        assert got.residue_pairs == g["matches"] and as_lists(got.pairs) == g["pairs"]
