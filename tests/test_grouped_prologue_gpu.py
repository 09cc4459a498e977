"""Grouped tables at the sizes where the prologue's block changes (a thread per problem, 32 to 1024, then
several problems a thread): the schedule is a permutation of the problems with the heaviest tiles first, its
prefix sums are the tiles of each problem, and the products are bit for bit the oracle's, on a second call
of the same plan too (tiles handed out by a counter, or one to a CTA)."""
import numpy as np
import pytest
import torch

import oracle
from gbblas import grouped
from gpu_util import assert_bit_equal, to_dev, to_host
from test_grouped_choice_gpu import f64_tiles

pytestmark = pytest.mark.gpu

F32_TILES = {1: (32, 32), 3: (64, 64)}


def tiles_and_work(dtype, cfg, m, n, k):
    if dtype == np.float64:
        tm, tn, fm, fn = f64_tiles(cfg, m, n)
        return tm * tn, fm * fn * max(k, 1)
    bm, bn = F32_TILES[cfg]
    return -(-m // bm) * -(-n // bn), min(m, bm) * min(n, bn) * max(k, 1)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 64, 65, 255, 257, 511, 513, 1023, 1024, 1025, 2050])
def test_block_sizes(cuda, count, dtype):
    g = np.random.default_rng(count)
    shapes = [tuple(int(x) for x in g.integers(1, 71 if i % 5 else 140, 3)) for i in range(count)]
    hs = [tuple(np.asfortranarray(g.uniform(-1, 1, s).astype(dtype)) for s in ((m, k), (k, n))) for m, n, k in shapes]
    Cs = [to_dev(np.full((m, n), np.nan, dtype)) for m, n, _ in shapes]
    plan = grouped.GroupedGemm([to_dev(a) for a, _ in hs], [to_dev(b) for _, b in hs], Cs)
    check = sorted({0, count - 1, *range(0, count, max(1, count // 60))})
    refs = {i: oracle.jmul(*hs[i], dtype=dtype) for i in check}
    for _ in range(2):
        for C in Cs:
            C.fill_(float("nan"))
        plan.run()
        torch.cuda.synchronize()
        assert not any(torch.isnan(C).any() for C in Cs)
        for i in check:
            assert_bit_equal(to_host(Cs[i]), refs[i])
        ws = plan.workspace.cpu().numpy()
        offsets = ws[:8 * (count + 1)].view(np.int64)
        words = ws[8 * (count + 1):][:4 * count].view(np.int32)
        order = [(int(w) & 0xFFFFFF, int(w) >> 24) for w in words]
        assert sorted(i for i, _ in order) == list(range(count))
        of = [tiles_and_work(dtype, cfg, *shapes[i]) for i, cfg in order]
        sums = np.concatenate([[0], np.cumsum([t for t, _ in of])])
        assert np.array_equal(offsets[1:], sums[1:])   # (the first word is the tile counter)
        buckets = [w.bit_length() for _, w in of]
        assert buckets == sorted(buckets, reverse=True)
