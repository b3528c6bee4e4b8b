"""sort_side's segment sort and its fallbacks against numpy's stable sort."""
import numpy as np
import pytest

from carmichael_frontier_b200 import mitm_gpu2 as G

CAP = 4096          # records of one segment


def keys_of(kind, n, rng):
    if kind == "uniform":
        return rng.integers(0, 3 << 51, n, dtype=np.uint64)
    if kind == "full":                       # up to 2^64 - 1, the largest key present
        k = rng.integers(0, 1 << 64, n, dtype=np.uint64)
        k[n // 2] = (1 << 64) - 1
        return k
    if kind == "small":                      # fewer values than bins: many equal keys
        return rng.integers(0, 1000, n, dtype=np.uint64)
    if kind == "equal":
        return np.full(n, 12345, dtype=np.uint64)
    if kind == "zero":
        return np.zeros(n, dtype=np.uint64)
    if kind == "clusters":                   # even segments whose records share a few bins
        c = rng.integers(0, 1 << 60, max(1, n // 100), dtype=np.uint64)
        return c[rng.integers(0, len(c), n)] + rng.integers(0, 2, n, dtype=np.uint64)
    if kind == "skewed":                     # nearly all keys in a small part of the range
        k = rng.integers(0, 1 << 20, n, dtype=np.uint64)
        k[0] = 1 << 62
        return k
    if kind == "products":                   # products of a few primes: spread over many powers of two
        return np.prod(rng.choice(np.array([3, 11, 29, 101, 331, 1009, 3001], dtype=np.uint64), (4, n)) +
                       2 * rng.integers(0, 500, (4, n), dtype=np.uint64), axis=0)
    if kind == "descending":
        return np.arange(n, 0, -1, dtype=np.uint64) << np.uint64(7)
    raise ValueError(kind)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uniform", "full", "small", "equal", "zero", "clusters", "skewed", "products", "descending"])
@pytest.mark.parametrize("n", [2, 33, CAP - 1, CAP, CAP + 1, 20_003, 65_536, 65_537, 3400 * 256, 3400 * 256 + 1, 3400 * 512 + 1, 5_000_011])
def test_sort_side_equals_numpy_stable_sort(cuda, kind, n):
    import torch
    rng = np.random.default_rng(n)
    k = keys_of(kind, n, rng)
    i = rng.integers(0, 1 << 63, n, dtype=np.uint64)
    dk, di = torch.from_numpy(k).to(cuda), torch.from_numpy(i).to(cuda)
    ok, oi = G.sort_side(dk, di)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(ok.cpu().numpy(), k[order]) and np.array_equal(oi.cpu().numpy(), i[order])
    assert np.array_equal(dk.cpu().numpy(), k) and np.array_equal(di.cpu().numpy(), i)   # inputs untouched


@pytest.mark.gpu
def test_sort_side_of_views_and_unaligned_slices(cuda):
    import torch
    rng = np.random.default_rng(7)
    k = rng.integers(0, 1 << 50, 100_001, dtype=np.uint64)
    dk = torch.from_numpy(k).to(cuda)
    ids = torch.arange(300_003, device=cuda, dtype=torch.int64).view(torch.uint64)
    for a, step in ((1, 1), (3, 1), (0, 2)):
        kk, ii = dk[a::step], ids[a:a + dk[a::step].numel()]
        ok, oi = G.sort_side(kk, ii)
        order = np.argsort(k[a::step], kind="stable")
        assert np.array_equal(ok.cpu().numpy(), k[a::step][order])
        assert np.array_equal(oi.cpu().numpy(), order.astype(np.uint64) + np.uint64(a))
