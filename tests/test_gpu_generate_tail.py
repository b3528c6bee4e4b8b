"""generate through the suffix table against the walker, and the merge join's tiles against numpy."""
import math
import random

import numpy as np
import pytest

from carmichael_frontier_b200 import mitm_gpu2 as G
from carmichael_frontier_b200.workloads import eligible_pool

MODULI = [2 ** 6 * 3 ** 3 * 5 ** 2 * 7 * 11 * 13 * 17 * 19, 2 ** 31 * 3 ** 4 * 5 * 7, 3 ** 5 * 5 ** 3 * 7 * 11, (1 << 62) - 2]


@pytest.mark.gpu
@pytest.mark.parametrize("r", range(3, 11))
@pytest.mark.parametrize("M", MODULI)
def test_suffix_table_records_equal_the_walkers(cuda, monkeypatch, r, M):
    primes = [p for p in eligible_pool(MODULI[0], 10 ** 4) if math.gcd(p, M) == 1]
    rng = random.Random(r)
    n = min(len(primes), 64 if r <= 10 else 16, {3: 64, 4: 64, 5: 40, 6: 30, 7: 26, 8: 24, 9: 22, 10: 22}[r])
    bits = 6
    total = math.comb(n, r)
    lo = rng.randrange(total // 2)
    hi = min(total, lo + 20_011)
    mult = rng.randrange(1, M)
    monkeypatch.setattr(G, "GEN_TAIL_MIN", 0)
    k, i = G.generate(primes[:n], r, M, mult, bits, lo, hi)
    monkeypatch.setattr(G, "GEN_TAIL_MIN", 1 << 60)
    k2, i2 = G.generate(primes[:n], r, M, mult, bits, lo, hi)
    assert np.array_equal(k.cpu().numpy(), k2.cpu().numpy()) and np.array_equal(i.cpu().numpy(), i2.cpu().numpy())
    for t in (0, (hi - lo) // 2, hi - lo - 1):
        idx = G.decode_ids(i[t:t + 1], r, bits)[0]
        assert int(k[t].item()) == mult * math.prod(primes[x] for x in idx) % M


@pytest.mark.gpu
@pytest.mark.parametrize("nD,nI", [(1, 1), (1, 5000), (5000, 1), (33, 2047), (1000, 2048), (4096, 2049), (100_000, 3000),
                                   (3000, 100_000), (50_000, 50_001)])
@pytest.mark.parametrize("values", [50, 10 ** 4, 10 ** 7, 10 ** 15])
def test_merge_join_equals_numpy(cuda, nD, nI, values):
    import torch
    if nD * nI / values > 3e6:
        pytest.skip("too many pairs")
    rng = np.random.default_rng(nD * 7 + nI)
    D = np.sort(rng.integers(0, values, nD, dtype=np.uint64))
    I = np.sort(rng.integers(0, values, nI, dtype=np.uint64))
    t = lambda a: torch.from_numpy(a).to(cuda)
    d, i = G.join_sorted(t(D), t(np.arange(nD, dtype=np.uint64)), t(I), t(np.arange(nI, dtype=np.uint64)))
    lo, hi = np.searchsorted(D, I, "left"), np.searchsorted(D, I, "right")
    ri = np.repeat(np.arange(nI), hi - lo)
    rd = np.concatenate([np.arange(a, b) for a, b in zip(lo, hi)]) if len(ri) else np.array([], dtype=int)
    assert np.array_equal(d.cpu().numpy(), rd.astype(np.uint64)) and np.array_equal(i.cpu().numpy(), ri.astype(np.uint64))
