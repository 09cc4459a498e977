"""FP64 products of more tiles than resident CTAs: every tile is computed once, whatever the remainder
after whole rounds, bit for bit; C is NaN before or folded in, so that a tile left out or done twice
shows."""
import numpy as np
import pytest
import torch

import gbblas
import oracle
from gpu_util import assert_bit_equal, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1000, 1000, 7), (608, 1024, 5), (1216, 512, 3), (1231, 517, 4), (2300, 1030, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_native_and_semiring_bit_exact(cuda, shape):
    M, N, K = shape
    g = np.random.default_rng(M + N + K)
    A, B, C = (np.asfortranarray(g.uniform(-1, 1, s)) for s in ((M, K), (K, N), (M, N)))
    Ad, Bd = to_dev(A), to_dev(B)
    Cd = to_dev(C)
    gbblas.gemm_(Cd, Ad, Bd, 1.5, 0.5)
    assert_bit_equal(to_host(Cd), oracle.gemm(A, B, C=C, alpha=1.5, beta=0.5))
    Cd = to_dev(np.full((M, N), np.nan))
    gbblas.jmul_(Cd, Ad, Bd)
    assert_bit_equal(to_host(Cd), oracle.jmul(A, B))
    Cd = to_dev(C)
    gbblas.gemm_semiring_(Cd, Ad, Bd, "min_plus", accumulate=True)
    torch.cuda.synchronize()
    assert_bit_equal(to_host(Cd), oracle.semiring_gemm(A, B, "min_plus", C=C, accumulate=True))
