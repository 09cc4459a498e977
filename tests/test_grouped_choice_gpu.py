"""The tile configuration that GB_GROUPED_AUTO gives each problem of a table, read back from the
schedule in the call's workspace (the order follows the count + 1 prefix sums: an int32 a problem, its
configuration in bits 24-30) and compared with the rules restated; results bit for bit either way."""
import numpy as np
import pytest
import torch

import oracle
from gbblas import grouped
from gpu_util import assert_bit_equal, to_dev, to_host

pytestmark = pytest.mark.gpu


def chosen(plan):
    """{problem: configuration} of the plan's last call."""
    torch.cuda.synchronize()
    words = plan.workspace.cpu().numpy()[8 * (plan.count + 1):][:4 * plan.count].view(np.int32)
    out = {int(w) & 0xFFFFFF: int(w) >> 24 for w in words}
    assert sorted(out) == list(range(plan.count))
    return [out[i] for i in range(plan.count)]


def run(shapes, dtype, check=True):
    g = np.random.default_rng(len(shapes) + shapes[0][0])
    hs = [tuple(np.asfortranarray(g.uniform(-1, 1, s).astype(dtype)) for s in ((m, k), (k, n))) for m, n, k in shapes]
    Cs = [to_dev(np.full((m, n), np.nan, dtype)) for m, n, _ in shapes]
    plan = grouped.GroupedGemm([to_dev(a) for a, _ in hs], [to_dev(b) for _, b in hs], Cs)
    plan.run()
    cfg = chosen(plan)
    if check:
        for (a, b), C in zip(hs, Cs):
            assert_bit_equal(to_host(C), oracle.jmul(a, b, dtype=dtype))
    return cfg


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def test_f32_line_is_three_quarters_of_a_piece_an_sm(cuda):
    line = sms() * 3072
    below, at = [(64, 48, 5)] * (sms() - 1) + [(64, 47, 5)], [(64, 48, 5)] * sms()
    assert sum(m * n for m, n, _ in at) == line
    assert run(below, np.float32) == [1] * len(below)
    assert run(at, np.float32) == [3] * len(at)
    assert run([(300, 300, 40)] * 16, np.float32) == [3] * 16
    assert run([(65, 65, 20)] * 50, np.float32) == [1] * 50


def f64_tiles(cfg, m, n):
    """(tiles down, tiles across, rows, columns) of a problem's equal tiles of at most 1024 elements."""
    bm, bn = {0: (16, 16), 1: (32, 32), 2: (64, 32), 3: (64, 32)}[cfg]
    tm = -(-m // bm)
    fm = -(-m // tm)
    tn = -(-n // min(bn, 1024 // fm))
    return tm, tn, fm, -(-n // tn)


def f64_load(tiles, k):
    tm, tn, fm, fn = tiles
    units = -(-fm * fn // 32)
    return tm * tn * (units * max(k, 1) + 26), -(-units // 4) * max(k, 1)


def f64_choice(shapes):
    """Per problem the cheapest of configurations 0-2 whose tiles the limit of 1024 elements does not
    narrow, or, below eight problems an SM, 0 for all when that ends sooner."""
    def whole(c, m, n):
        return c < 2 or f64_tiles(c, m, n)[1] == -(-n // 32)

    best = [min((c for c in range(3) if whole(c, m, n)), key=lambda c: (f64_load(f64_tiles(c, m, n), k)[0], c))
            for m, n, k in shapes]
    if len(shapes) >= 8 * sms():
        return best

    def time(cfgs):
        loads = [f64_load(f64_tiles(c, m, n), k) for c, (m, n, k) in zip(cfgs, shapes)]
        return max(sum(t for t, _ in loads), max(l for _, l in loads) * 4 * sms())

    return [0] * len(shapes) if time([0] * len(shapes)) < time(best) else best


@pytest.mark.parametrize("shapes", [[(100, 100, 100)], [(64, 64, 64)] * 10, [(100, 100, 30)] * 64, [(33, 17, 65)] * 300,
                                    [(16, 16, 16)] * 40, [(61, 47, 2), (1, 1, 1), (64, 64, 200)], [(200, 3, 9)] * 700],
                         ids=lambda s: "%dx%s" % (len(s), s[0]))
def test_f64_choice(cuda, shapes):
    assert run(shapes, np.float64) == f64_choice(shapes)


@pytest.mark.parametrize("count,hi", [(20, 130), (150, 90), (700, 64), (3000, 40)])
def test_f64_choice_of_uneven_tables(cuda, count, hi):
    g = np.random.default_rng(count)
    shapes = [tuple(int(x) for x in np.rint(np.exp(g.uniform(0, np.log(hi), 3)))) for _ in range(count)]
    assert run(shapes, np.float64, check=count < 1000) == f64_choice(shapes)


def test_f64_tiles_of_explicit_configurations(cuda):
    shapes = [(64, 64, 5), (61, 47, 9), (100, 100, 7), (65, 33, 3), (130, 17, 6), (2, 200, 4), (40, 64, 2)]
    g = np.random.default_rng(3)
    hs = [tuple(np.asfortranarray(g.uniform(-1, 1, s)) for s in ((m, k), (k, n))) for m, n, k in shapes]
    for cfg in range(4):
        Cs = [to_dev(np.full((m, n), np.nan)) for m, n, _ in shapes]
        plan = grouped.GroupedGemm([to_dev(a) for a, _ in hs], [to_dev(b) for _, b in hs], Cs,
                                   tuning=grouped.Tuning.from_list([cfg] * grouped.CLASSES))
        plan.run()
        assert chosen(plan) == [cfg] * len(shapes)
        for (a, b), C in zip(hs, Cs):
            assert_bit_equal(to_host(C), oracle.jmul(a, b))
        offsets = plan.workspace.cpu().numpy()[:8 * (plan.count + 1)].view(np.int64)
        assert offsets[-1] == sum(f64_tiles(cfg, m, n)[0] * f64_tiles(cfg, m, n)[1] for m, n, _ in shapes)
