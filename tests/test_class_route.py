"""Which instances take the class join: decided on the host, so tested without a GPU."""
import math
import os

import numpy as np
import pytest

from carmichael_frontier_b200 import Instance, Solver, Tuning, _lib
from carmichael_frontier_b200.portfolio import BatchSolver, BatchTuning
from carmichael_frontier_b200.solve import _ws_bytes
from carmichael_frontier_b200.workloads import eligible_pool

M = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19 * 23 * 29
Q = eligible_pool(M, 10 ** 5)
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def instance(k, n, r):
    return Instance.build(M, Q[:k + n], Q[:k], r, math.prod(Q[:k]) * 10 ** 8)


def class_plan(x, **tuning):
    s = Solver("cuda", tuning=Tuning(**tuning))
    nD, nI = math.comb(len(x.B0), x.r), math.comb(len(x.INS), x.r)
    return s._class_plan(x, s.plan(nD, nI))


@pytest.mark.parametrize("side", ["B0", "INS"])
def test_primes_of_2_31_or_more_do_not_take_the_class_join(side):
    # its kernels multiply 32-bit factors; Instance.build refuses such primes, the class itself does not
    x = instance(64, 150, 4)
    assert class_plan(x) is not None
    getattr(x, side)[-1] = (1 << 31) + 11
    x.P0 = math.prod(x.B0)
    assert class_plan(x) is None


def test_workspaces_above_the_limit_are_declined():
    x = instance(64, 160, 5)
    need = _ws_bytes(class_plan(x))
    assert class_plan(x, class_ws_bytes=need) is not None and class_plan(x, class_ws_bytes=need - 1) is None
    big = instance(64, 155, 6)                     # 1.5e10 I records: 10 GB, the table join 1.4
    assert _ws_bytes(class_plan(big)) > 8 << 30 and class_plan(big, class_ws_bytes=8 << 30) is None
    s = Solver("cuda", tuning=Tuning(class_ws_bytes=2 * need - 1))
    plan = s.plan(math.comb(64, 5), math.comb(160, 5))
    assert s._class_plan(x, plan) is not None
    s._pool = object()                             # in a list: two workspaces are held
    assert s._class_plan(x, plan) is None
    for budget, taken in ((2 * need, True), (2 * need - 1, False)):
        b = BatchSolver("cuda", tuning=BatchTuning(mem_budget=budget))
        assert (b._class_plan(x, math.comb(64, 5), math.comb(160, 5), None) is not None) == taken


EXHAUSTED = """
import ctypes as C, resource, sys
from carmichael_frontier_b200 import _lib
lib = _lib.load()
libc = C.CDLL(None)
libc.malloc.restype = C.c_void_p
libc.malloc.argtypes = [C.c_size_t]
n = lib.cf_class_plan_bytes()
out = C.create_string_buffer(n)
at, m, i_n = C.addressof(out), %d, %d
assert lib.cf_class_plan(m, 64, 120, 4, 0, i_n, 0, at, n) == _lib.CF_OK
assert lib.cf_class_plan(m, 0, 120, 4, 0, i_n, 0, at, n) == _lib.CF_EBADARG   # this thread's error text exists
pages = int(open("/proc/self/statm").read().split()[0])
resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize(),) * 2)
for size in (1 << 20, 1 << 12, 256, 64, 16):
    while libc.malloc(size):
        pass
rc = lib.cf_class_plan(m, 64, 120, 4, 0, i_n, 0, at, n)
sys.stdout.write("status %%d" %% rc)
"""


def test_a_plan_without_host_memory_returns_a_status():
    # an exception that leaves a C function ends the process
    import subprocess
    import sys
    p = subprocess.run([sys.executable, "-c", EXHAUSTED % (M // (M & -M), math.comb(120, 4))], capture_output=True,
                       text=True, cwd=ROOT, timeout=120)
    if "MemoryError" in p.stderr:
        pytest.skip("the interpreter itself had no memory left")
    assert p.returncode == 0 and p.stdout in (f"status {_lib.CF_OK}", f"status {_lib.CF_ENOMEM}"), (p.returncode, p.stderr[-500:])


def test_small_probing_sides_keep_the_table_join_at_small_radii():
    for k, n, r, taken in ((64, 102, 4, False), (64, 120, 4, False), (64, 140, 4, True), (64, 200, 3, False),
                           (100, 440, 3, True), (104, 12, 4, True), (104, 30, 4, False), (64, 58, 5, True), (30, 58, 5, True)):
        assert max(math.comb(k, r), math.comb(n, r)) >= 1 << 20
        assert (class_plan(instance(k, n, r)) is not None) == taken, (k, n, r)


def test_portfolio_batches_small_probing_sides_where_there_is_a_batch(monkeypatch):
    # nothing is launched here: the split is made before the tables go up
    class Split(Exception):
        pass

    def stop(*a):
        raise Split(a[0])

    import carmichael_frontier_b200.portfolio as P
    for counts, batched in (((5, 0, 2), 0), ((8, 0, 2), 8), ((1, 1, 1), 2), ((1, 0, 0), 0)):
        xs = [instance(64, 110, 4)] * counts[0] + [instance(20, 30, 3)] * counts[1] + [instance(64, 60, 5)] * counts[2]
        seen = []
        monkeypatch.setattr(P, "pool_table_host", lambda *a: seen.append(a) or np.zeros(8, dtype=np.uint8))
        monkeypatch.setattr(P, "screen_table_host", lambda *a: np.zeros(8, dtype=np.uint8))
        b = BatchSolver("cuda")
        monkeypatch.setattr(b, "torch", type("T", (), {"from_numpy": staticmethod(stop)}))
        with pytest.raises(Split):
            b.prepare(xs)
        assert len(seen) == 2 * batched


def solve_status(x, cp, pD=None, pI=None, **other):
    """(status, error text) of cf_solve with a class plan.  The device addresses are never used by a call that
    is refused."""
    import ctypes as C
    lib = _lib.load()
    pD = np.array(x.B0, dtype=np.uint64) if pD is None else pD
    pI = np.array(x.INS, dtype=np.uint64) if pI is None else pI
    lb = np.ones(1, dtype=np.uint32)
    stage = np.zeros(lib.cf_solve_table_bytes(len(pD), len(pI), x.r), dtype=np.uint8)
    args = dict(primesD=pD.ctypes.data, primesI=pI.ctypes.data, m=M // (M & -M), multD_odd=1, multD_2=1, n_D=1,
                n_I=math.comb(len(pI), x.r), limbsB=lb.ctypes.data, nlimbs=1, lgP0=1.0, lgB=1.0, eps=1e-6, nD=len(pD),
                nI=len(pI), r=x.r, a=6, class_plan=C.cast(C.c_char_p(cp), C.c_void_p), stage=stage.ctypes.data, tables=256,
                ws=256, ws_bytes=1 << 62, misc=256)
    rc = lib.cf_solve(C.byref(_lib.CfSolve(**{**args, **other})), None)
    assert not stage.any()
    return rc, lib.cf_last_error_string()


def test_cf_solve_refuses_a_class_plan_for_primes_of_2_31_or_more():
    x = instance(64, 150, 4)
    for big in (0, 1):
        sides = [np.array(x.B0, dtype=np.uint64), np.array(x.INS, dtype=np.uint64)]
        sides[big][-1] = (1 << 31) + 11
        rc, text = solve_status(x, class_plan(x), *sides)
        assert rc == _lib.CF_EBADARG and b"2^31" in text


@pytest.mark.parametrize("what", ["smaller I pool", "larger D pool", "radius", "window", "start", "swap", "modulus"])
def test_cf_solve_refuses_the_plan_of_another_instance(what):
    x = instance(64, 150, 4)
    cp, y, other = class_plan(x), x, {}
    if what == "smaller I pool":
        y = instance(64, 149, 4)
        other = dict(n_I=math.comb(150, 4))
    elif what == "larger D pool":
        y = instance(65, 150, 4)
    elif what == "radius":
        other = dict(r=5)
    elif what == "window":
        other = dict(n_I=math.comb(150, 4) - 1)
    elif what == "start":
        other = dict(i_lo=1)
    elif what == "swap":
        other = dict(swap=1)
    else:
        other = dict(m=3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 31)      # without divisors of the plan
    rc, text = solve_status(y, cp, **other)
    assert rc == _lib.CF_EBADARG and b"another instance" in text
