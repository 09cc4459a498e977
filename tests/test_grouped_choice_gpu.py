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
