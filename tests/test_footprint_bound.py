"""serve.footprint is an upper bound on what a solve holds, class join included."""
import math

import numpy as np
import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning, serve
from carmichael_frontier_b200.bsolve import BoundedSolve
from carmichael_frontier_b200.solve import class_pairs
from carmichael_frontier_b200.workloads import eligible_pool

M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
Q = eligible_pool(M, 10 ** 5)


def instance(k, n, r, slack):
    return Instance.build(M, Q[:k + n], Q[:k], r, math.prod(Q[:k]) * slack)


@pytest.mark.parametrize("strategy", ["fused", "auto"])
def test_pair_buffers_and_the_workspace_limit_are_counted(strategy):
    x = instance(64, 150, 6, 10 ** 9)                  # 2^20 pair and result rows: 109 MB beside the workspace
    tu = Tuning(strategy=strategy)
    rows = 104 * class_pairs(math.comb(64, 6), math.comb(150, 6), M, tu)
    assert rows > 100 << 20
    declined = serve.footprint(x, Tuning(strategy=strategy, class_join=False))["bytes"]
    ws = serve.footprint(x, tu)["bytes"] - rows - (64 << 20)
    assert 6 << 30 < ws < 24 << 30 or ws + (64 << 20) == declined     # the larger of the two joins
    assert serve.footprint(x, Tuning(strategy=strategy, class_ws_bytes=1 << 30))["bytes"] == declined


@pytest.mark.gpu
@pytest.mark.parametrize("r,n,slack,strategy", [(5, 150, 10 ** 9, "fused"), (5, 100, 10 ** 9, "fused"),
                                                (4, 170, 10 ** 4, "auto"), (5, 90, 10 ** 4, "auto")])
@pytest.mark.parametrize("overflow", [False, True])
def test_a_solve_holds_no_more_than_its_footprint(cuda, monkeypatch, r, n, slack, strategy, overflow):
    import torch
    x = instance(64, n, r, slack)
    tu = Tuning(strategy=strategy)
    if overflow:                                       # one chunk of survivors: the other join after the class join
        real = Solver._class_plan

        def short(self, inst, plan):
            p = real(self, inst, plan)
            if p is None:
                return None
            a = np.frombuffer(p, dtype=np.uint32).copy()
            a[18] = 1
            return a.tobytes()

        monkeypatch.setattr(Solver, "_class_plan", short)
    s = Solver(cuda, tuning=tu)
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    res = s.solve_instance(x)
    peak = torch.cuda.max_memory_allocated() - base
    fp = serve.footprint(x, tu)
    assert peak <= fp["bytes"]
    by_class = res.plan.get("table") == "class" or bool(res.plan.get("class_plan"))
    assert by_class == (not overflow)
    del res
