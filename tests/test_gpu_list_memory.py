"""A list of uneven pools finds its buffers when its first solve is queued."""
import math

import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning
from carmichael_frontier_b200.workloads import draw_modulus, eligible_pool

pytestmark = pytest.mark.gpu


def instances(pools, k, r):
    out, seed = [], 1
    for pool in pools:
        while True:
            M = draw_modulus(seed)
            Q = eligible_pool(M, 10 ** 5)
            seed += 1
            if len(Q) >= pool:
                break
        out.append(Instance.build(M, Q[:pool], Q[:k], r, math.prod(Q[:k]) * 10 ** 8))
    return out


@pytest.mark.parametrize("pools,k,r,tu", [
    ((124, 214, 140, 200, 130, 180, 208, 160), 64, 5, Tuning()),
    ((124, 190, 140, 214, 130, 180, 208, 160), 64, 4, Tuning(class_min_probe=0)),
    ((90, 140, 70, 120, 200, 100), 30, 3, Tuning(class_join=False))])
def test_no_buffer_grows_inside_a_list(cuda, monkeypatch, pools, k, r, tu):
    import torch
    insts = instances(pools, k, r)
    s = Solver(cuda, tuning=tu)
    seen = []
    real = Solver.enqueue

    def enqueue(self, inst, plan, marks=None):
        if not seen:
            seen.append(torch.cuda.memory_stats()["segment.all.allocated"])
            seen.append({k: t.data_ptr() for k, t in self._bufs.items()})
            seen.append({k: t.data_ptr() for k, (t, _) in self._pinned.items()})
        return real(self, inst, plan, marks)

    monkeypatch.setattr(Solver, "enqueue", enqueue)
    out = s.solve_many(insts)
    assert torch.cuda.memory_stats()["segment.all.allocated"] == seen[0]
    assert {k: t.data_ptr() for k, t in s._bufs.items()} == seen[1]
    assert {k: t.data_ptr() for k, (t, _) in s._pinned.items()} == seen[2]
    monkeypatch.undo()
    for x, a in zip(insts[:3], out):
        b = Solver(cuda, tuning=tu).solve_instance(x)
        assert (a.residue_pairs, a.pairs, a.n_I) == (b.residue_pairs, b.pairs, b.n_I)
