"""Which tiles of a term product or an adjoint on CTA pairs are cut along K, and what that leaves alone.
A launch on single CTAs never cuts and gives whole tiles the same bits, so whole tiles are equal there
and every cut tile differs somewhere (its sums are rounded in another order): with whole tiles before the
cut ones, with C folded in, with a remainder that spans both halves of an adjoint, and not at all where
the parts would cost more than they save."""
import math

import numpy as np
import pytest
import torch

import gbblas
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


def raster(t, tiles_m, tiles_n, band=8):
    """(row, column) of tile t."""
    b, at = divmod(t, band * tiles_n)
    rows = min(band, tiles_m - b * band)
    return b * band + at % rows, at // rows


def plan(tiles, panels, terms, pairs):
    """(first cut tile, parts), parts = 1 for none: the cost rule restated."""
    total = sum(tiles)
    cuts = total % pairs
    first = total - cuts
    least, once, part = (0.8, 20, 7) if first else (0.75, 32, 2)
    seen = [p for t, p, end in zip(tiles, panels, np.cumsum(tiles)) if t and end > first]
    share = lambda n: terms * math.ceil(max(seen) / n) * max(n * cuts / pairs, least)   # noqa: E731
    cost = {1: share(1)} if cuts else {1: 0.0}
    for n in range(2, min(seen) + 1):
        if n * cuts <= pairs and cuts:
            cost[n] = share(n) + once + part * (n - 2)
    best = min(cost, key=lambda n: (cost[n], n))
    return first, best


def both_engines(call):
    out = []
    for engine in (2, 1):
        gbblas.set_tc_engine(engine)
        try:
            out.append(call())
            torch.cuda.synchronize()
            gbblas.check_device_status()
        finally:
            gbblas.set_tc_engine(0)
    return out


def check(pair, single, tiles_m, tiles_n, start, first, parts):
    for t in range(tiles_m * tiles_n):
        i, j = raster(t, tiles_m, tiles_n)
        s = (slice(256 * i, 256 * i + 256), slice(256 * j, 256 * j + 256))
        same = np.array_equal(pair[s].view(np.uint32), single[s].view(np.uint32))
        assert same == (parts == 1 or start + t < first), (t, first, parts)


@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("case", [("bf16x6", 1600, 3328, 1312), ("bf16x3", 1600, 3328, 1312), ("bf16x6", 2304, 2300, 2000),
                                  ("bf16x3", 2304, 2300, 2000), ("bf16x6", 700, 300, 3001), ("bf16x6", 1024, 1024, 1024),
                                  ("bf16x6", 20000, 100, 700), ("bf16x6", 20000, 100, 400), ("bf16x3", 3001, 2503, 300)],
                         ids=lambda c: "%s-%dx%dx%d" % c)
def test_term_products(cuda, case, beta):
    mode, M, N, K = case
    tm, tn = -(-M // 256), -(-N // 256)
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    first, parts = plan([tm * tn], [-(-K // 64)], 3 if mode == "bf16x3" else 6, pairs)
    if pairs == 76:   # the shapes keep standing for what they were chosen for
        assert (parts > 1) == (case[1:] not in ((20000, 100, 400), (3001, 2503, 300)))
        assert (first > 0) == (M not in (700, 1024))
    g = np.random.default_rng(M + K)
    A, B, C = (to_dev(g.standard_normal(s).astype(np.float32)) for s in ((M, K), (K, N), (M, N)))

    def call():
        out = C.clone(memory_format=torch.preserve_format)
        return to_host(gbblas.gemm_(out, A, B, 1.5, beta, mode=mode) if beta else
                       gbblas.gemm_(out, A, B, mode=mode))

    pair, single = both_engines(call)
    check(pair, single, tm, tn, 0, first, parts)


@pytest.mark.parametrize("shape", [(2304, 256, 2300), (700, 520, 300), (2816, 300, 1500)],
                         ids=lambda s: "x".join(map(str, s)))
def test_adjoint(cuda, shape):
    M, N, K = shape
    t = lambda x: -(-x // 256)   # noqa: E731
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    tiles = [t(M) * t(K), t(K) * t(N)]
    first, parts = plan(tiles, [-(-N // 64), -(-M // 64)], 3, pairs)
    if pairs == 76 and shape == (2304, 256, 2300):
        assert parts > 1 and 0 < first < tiles[0]   # the remainder spans dA and dB
    g = np.random.default_rng(M)
    A, B, W = (to_dev(g.standard_normal(s).astype(np.float32)) for s in ((M, K), (K, N), (M, N)))

    def call():
        dA = torch.full((K, M), float("nan"), dtype=torch.float32, device="cuda").t()
        dB = torch.full((N, K), float("nan"), dtype=torch.float32, device="cuda").t()
        gbblas.gemm_adjoint_(dA, dB, A, B, W)
        return to_host(dA), to_host(dB)

    (dA2, dB2), (dA1, dB1) = both_engines(call)
    check(dA2, dA1, t(M), t(K), 0, first, parts)
    check(dB2, dB1, t(K), t(N), tiles[0], first, parts)
