"""The ways an FP64 tile stores C (the chain as it is, scaled, with C folded in): each alpha and beta
that tells them apart, zeros of both signs included, at tiles of one to eight elements a lane and ragged
ends, native and grouped; with beta = 0 of either sign C is not read (NaN before)."""
import numpy as np
import pytest
import torch

import gbblas
import oracle
from gbblas import grouped
from gpu_util import assert_bit_equal, to_dev, to_host

pytestmark = pytest.mark.gpu

AB = [(1.0, 0.0), (1.0, -0.0), (-1.0, 0.0), (0.75, -0.0), (1.0, 1.0), (-1.5, 0.5), (1.0, 5e-324), (5e-324, 2.0)]
SHAPES = [(1, 1, 3), (8, 8, 5), (16, 16, 3), (33, 17, 4), (64, 16, 9), (61, 29, 2), (500, 470, 3)]


def _operands(shape, beta):
    M, N, K = shape
    g = np.random.default_rng(M * N + K)
    A, B, C = (np.asfortranarray(g.uniform(-1, 1, s)) for s in ((M, K), (K, N), (M, N)))
    return A, B, (C if beta != 0.0 else np.asfortranarray(np.full((M, N), np.nan)))


@pytest.mark.parametrize("ab", AB, ids=str)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_native(cuda, shape, ab):
    A, B, C = _operands(shape, ab[1])
    Cd = to_dev(C)
    gbblas.gemm_(Cd, to_dev(A), to_dev(B), *ab)
    ref = oracle.gemm(A, B, C=C if ab[1] != 0.0 else None, alpha=ab[0], beta=ab[1] if ab[1] != 0.0 else 0.0)
    assert_bit_equal(to_host(Cd), ref)


@pytest.mark.parametrize("config", [0, 1, 2, 3, grouped.AUTO])
def test_grouped(cuda, config):
    cases = [(s, ab) + _operands(s, ab[1]) for s in SHAPES for ab in AB]
    Cs = [to_dev(c[4]) for c in cases]
    plan = grouped.GroupedGemm([to_dev(c[2]) for c in cases], [to_dev(c[3]) for c in cases], Cs,
                               [c[1][0] for c in cases], [c[1][1] for c in cases],
                               tuning=grouped.Tuning.from_list([config] * grouped.CLASSES))
    plan.run()
    torch.cuda.synchronize()
    for (s, ab, A, B, C), Cd in zip(cases, Cs):
        ref = oracle.gemm(A, B, C=C if ab[1] != 0.0 else None, alpha=ab[0], beta=ab[1] if ab[1] != 0.0 else 0.0)
        assert_bit_equal(to_host(Cd), ref)
