"""cf_gen_subsets_tail called directly: rank ranges past the last subset, pools without a suffix table."""
import math

import pytest

from carmichael_frontier_b200 import _lib
from carmichael_frontier_b200.tables import pool_table_host
from carmichael_frontier_b200.workloads import eligible_pool


def test_ranks_past_the_last_subset_are_refused():
    # refused on the host, before anything is read: the addresses are never used
    lib = _lib.load()
    for n, r in ((9, 3), (64, 5), (1024, 10)):
        total = min(math.comb(n, r), (1 << 64) - 1)
        for lo, count in ((total - 1, 2), (total, 1), (total + 7 & (1 << 64) - 1, 1), (0, total + 1), ((1 << 64) - 1, 1 << 39)):
            if lo + count <= total or count > 1 << 40 or count < 1:
                continue
            rc = lib.cf_gen_subsets_tail(256, 256, n, r, lo, count, 1, 0, 1, 256, 256, None, None)
            assert rc == _lib.CF_EBADARG and b"C(n, r)" in lib.cf_last_error_string(), (n, r, lo, count)


SMOOTH = 2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19


@pytest.mark.gpu
@pytest.mark.parametrize("r", [3, 4, 7, 10])
@pytest.mark.parametrize("M,big,ok", [(SMOOTH, False, True), (SMOOTH, True, False), (3 ** 4 * 5 << 33, False, False)])
def test_pools_without_a_suffix_table_are_reported(cuda, r, M, big, ok):
    import torch
    lib = _lib.load()
    primes = [p for p in eligible_pool(SMOOTH, 10 ** 4) if math.gcd(p, M) == 1][:r + 7]
    if big:
        primes[-1] = (1 << 61) - 1
    n = len(primes)
    pool = torch.from_numpy(pool_table_host(primes, r, M, 12345)).to(cuda)
    tail = torch.zeros(max(16, lib.cf_tail_bytes(n, r)), dtype=torch.uint8, device=cuda)
    _lib.check(lib.cf_build_tail(pool.data_ptr(), n, r, tail.data_ptr(), _lib.stream_handle()), "cf_build_tail")
    lo, count = 5, math.comb(n, r) - 5
    got = torch.full((2, count), -1, dtype=torch.int64, device=cuda)
    want = torch.zeros(2, count, dtype=torch.int64, device=cuda)
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    _lib.check(lib.cf_gen_subsets_tail(pool.data_ptr(), tail.data_ptr(), n, r, lo, count, 0, 6, 1, got[0].data_ptr(),
                                       got[1].data_ptr(), err.data_ptr(), _lib.stream_handle()), "tail")
    _lib.check(lib.cf_gen_subsets(pool.data_ptr(), n, r, lo, count, 0, 6, 1, want[0].data_ptr(), want[1].data_ptr(),
                                  _lib.stream_handle()), "walker")
    assert err.item() == (0 if ok else _lib.ERR_BAD_ARG)
    assert torch.equal(got, want) if ok else bool((got == -1).all())
