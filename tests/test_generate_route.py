"""Which generate() calls use the pool's suffix table: the library and the device tables are stand-ins here."""
import math

import pytest

from carmichael_frontier_b200 import mitm_gpu2 as G
from carmichael_frontier_b200.workloads import draw_modulus, eligible_pool


@pytest.mark.parametrize("r,n,count,tail", [
    (3, 320, 5_000_000, False), (3, 64, 1 << 15, False), (4, 120, 1 << 17, False), (4, 120, (1 << 22) - 1, False),
    (4, 120, 1 << 22, True), (5, 70, 1 << 17, False), (5, 70, 1 << 18, True), (6, 40, (1 << 17) - 1, False),
    (6, 40, 1 << 17, True), (7, 40, 1 << 20, True), (2, 500, 100_000, False)])
def test_route(monkeypatch, r, n, count, tail):
    import torch

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append(name) or 0

    class Tables:
        pool = tail = lambda self, *a: torch.empty(0)

    calls = []
    M = draw_modulus(40)
    primes = eligible_pool(M, 10 ** 5)
    primes = (primes + [p for p in range(10 ** 5, 3 * 10 ** 5) if math.gcd(p, M) == 1])[:n]
    real = torch.empty
    monkeypatch.setattr(G, "_device", lambda d: torch.device("cpu"))
    monkeypatch.setattr(G, "_dtables", lambda d: Tables())
    monkeypatch.setattr(G._lib, "load", lambda: Lib())
    monkeypatch.setattr(G._lib, "stream_handle", lambda *a: 0)
    monkeypatch.setattr(torch, "empty", lambda *a, **k: real(1, dtype=k.get("dtype")))
    G.generate(primes, r, M, 1, 10 if r < 7 else 6, 0, count)
    assert calls == ["cf_gen_subsets_tail" if tail else "cf_gen_subsets"]
