"""sort_side on keys that the segment sort's map has to find first: narrow ranges, ordered input, uneven
keys sampled thinly, a dense piece cut by the largest key, few distinct keys -- results and route."""
import numpy as np
import pytest

from carmichael_frontier_b200 import _lib
from carmichael_frontier_b200 import mitm_gpu2 as G

pytestmark = pytest.mark.gpu
CAP = 4096


def keys_of(kind, n, rng):
    u64 = np.uint64
    if kind.startswith("narrow"):                  # even keys below a bound near or below the number of bins
        return rng.integers(0, int(kind[6:]), n, dtype=u64)
    if kind == "ascending":
        return np.arange(n, dtype=u64) << u64(20)
    if kind == "ascending runs":                   # 16 ordered runs one after another
        return np.sort(rng.integers(0, 3 << 51, n, dtype=u64).reshape(16, -1) if n % 16 == 0 else
                       rng.integers(0, 3 << 51, n, dtype=u64)).ravel()
    if kind == "products":                         # small products far below the largest: thin pieces
        return np.prod(rng.integers(3, 1 << 13, (4, n), dtype=u64), axis=0)
    if kind == "cut":                              # a tenth of the records low, the rest even up to a bound inside a piece;
        k = rng.integers(0, (1 << 50) + (1 << 44), n, dtype=u64)
        low = rng.random(n) < 0.1                  # the low ones end inside a piece too, which no piece's share shows
        k[low] >>= u64(9)
        return k
    if kind == "smooth cut":                       # the low ones thin out instead
        k = rng.integers(0, (1 << 50) + (1 << 44), n, dtype=u64)
        low = rng.random(n) < 0.1
        k[low] = (k[low] * rng.random(low.sum()) ** 4).astype(u64)
        return k
    if kind == "pairs":                            # ordered, every key twice
        return np.arange(n, dtype=u64) // u64(2) << u64(9)
    if kind.startswith("few"):                     # that many distinct keys over 50 bits
        return rng.integers(0, 1 << 50, int(kind[3:]), dtype=u64)[rng.integers(0, int(kind[3:]), n)]
    if kind == "one":
        return np.full(n, (1 << 64) - 1, dtype=u64)
    raise ValueError(kind)


def sort(cuda, k, i):
    """(keys, ids, whether the segment sort held) of cf_sort_pairs_to with a workspace of its own.  The
    control words behind the second buffers and the map are as the segment sort left them, or the LSD sort
    has written over them."""
    import torch
    lib = _lib.load()
    n = len(k)
    dk, di = torch.from_numpy(k).to(cuda), torch.from_numpy(i).to(cuda)
    ko, io = torch.empty_like(dk), torch.empty_like(di)
    nb = lib.cf_sort_to_tmp_bytes(n)
    tmp = torch.empty(nb, dtype=torch.uint8, device=cuda)
    _lib.check(lib.cf_sort_pairs_to(dk.data_ptr(), di.data_ptr(), ko.data_ptr(), io.data_ptr(), n, 8, tmp.data_ptr(), nb,
                                    _lib.stream_handle()), "sort")
    assert tmp.data_ptr() % 256 == 0
    at = -(-2 * 8 * (n + (n & 1)) // 256) * 256 + 4 * (3 * 2048 + 2)
    top, _mode, _met, seg, _err, bail = tmp[at + 24:at + 48].cpu().numpy().view(np.uint32).tolist()
    return ko.cpu().numpy(), io.cpu().numpy(), top == (-(-n // 3400) << 13) - 1 and seg <= CAP and bail == 0


@pytest.mark.parametrize("kind,n,held", [
    ("narrow1000", 20_003, True), ("narrow1048576", 1 << 20, True), ("narrow1048576", 7_624_512, True),
    ("narrow16777216", (1 << 24) + 7, True), ("narrow5000000", 4_000_001, True), ("narrow65536", 65_537, True),
    ("ascending", 20_003, True), ("ascending", 1 << 22, True), ("ascending", 20_000_003, True),
    ("ascending runs", 1 << 24, True), ("pairs", 5_000_001, True),
    ("products", 7_624_512, True), ("products", 30_000_001, True), ("cut", 1 << 20, True), ("cut", 20_000_001, False),
    ("smooth cut", 1 << 20, True), ("smooth cut", 7_624_512, True), ("smooth cut", 20_000_001, True),
    ("cut", 65_000, True), ("few1000", 1 << 20, False), ("few1000", 7_624_512, False), ("few70000", 7_624_512, False),
    ("few100", 65_537, True), ("few2000000", 7_624_512, True), ("few400000", 7_624_512, False),
    ("few3", 20_003, False), ("one", 20_003, True), ("one", 65_536, True), ("one", 65_537, False), ("one", 3_000_000, False)])
def test_sort_and_its_route(cuda, kind, n, held):
    rng = np.random.default_rng(n)
    k = keys_of(kind, n, rng)
    i = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    ko, io, got = sort(cuda, k, i)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(ko, k[order]) and np.array_equal(io, i[order])
    assert got == held
