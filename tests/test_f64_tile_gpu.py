"""The FP64 tiles whose elements are dealt to the warps 32 at a time: native and kernel! products at
the edges of the tile shapes (16, 32, 64 rows; 8, 16, 32 columns; panels of 8, 16 and 32 k), with
padded leading dimensions, every orientation and alpha / beta, and grouped products under the FP64
tile choices.  All bit-identical to the oracle's FMA chain."""
import numpy as np
import pytest
import torch

import gbblas
import oracle
from gbblas import grouped
from gpu_util import assert_bit_equal, to_dev, to_dev_ld, to_host

pytestmark = pytest.mark.gpu

# 1 and 33 past a shape's edge; one tile, one tile per SM, several; K around each panel length
SHAPES = [(1, 1, 1), (1, 300, 9), (300, 1, 33), (16, 16, 32), (17, 16, 31), (16, 17, 33), (32, 32, 16), (33, 32, 17),
          (64, 16, 8), (65, 33, 7), (31, 129, 64), (400, 390, 24), (611, 613, 40), (1100, 1000, 19)]


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_native_edges_bit_exact(cuda, shape, trans):
    M, N, K = shape
    ta, tb = trans
    g = np.random.default_rng(M * 31 + N * 17 + K + 2 * ta + tb)
    A = g.uniform(-1, 1, (K, M) if ta else (M, K))
    B = g.uniform(-1, 1, (N, K) if tb else (K, N))
    C = g.uniform(-1, 1, (M, N))
    for alpha, beta in ((1.0, 0.0), (1.5, 0.5)):
        ref = oracle.gemm(np.asfortranarray(A), np.asfortranarray(B), C=np.asfortranarray(C), alpha=alpha, beta=beta,
                          trans_a=bool(ta), trans_b=bool(tb))
        Av, _ = to_dev_ld(A, A.shape[0] + 3)   # NaN in the padding of A and B
        Bv, _ = to_dev_ld(B, B.shape[0] + 1)
        Cv, Cbuf = to_dev_ld(C, M + 2, fill=7.0)
        gbblas.gemm_raw(ta, tb, M, N, K, alpha, Av.data_ptr(), A.shape[0] + 3, Bv.data_ptr(), B.shape[0] + 1, beta,
                        Cv.data_ptr(), M + 2, dtype=torch.float64, stream=torch.cuda.current_stream().cuda_stream)
        assert_bit_equal(to_host(Cv), ref)
        assert np.all(to_host(Cbuf)[M:, :] == 7.0)


@pytest.mark.parametrize("shape", [(1, 1, 5), (16, 16, 32), (33, 65, 17), (200, 190, 40)])
def test_kernel_edges_bit_exact(cuda, shape):
    M, N, K = shape
    g = np.random.default_rng(M + N + K)
    D, A, X = g.uniform(-1, 1, (M, N)), g.uniform(-1, 1, (M, K)), g.uniform(-1, 1, (K, N))
    Dd = to_dev(D)
    gbblas.kernel_(Dd, to_dev(A), to_dev(X))
    ref = oracle.kernel_chain(D.ravel(order="F"), A.ravel(order="F"), X.ravel(order="F"), M, N, M, K, K)
    assert_bit_equal(to_host(Dd).ravel(order="F"), ref)


def test_signed_zeros_infinities_and_nan(cuda):
    """-0 chains, Inf * 0 and NaN reach only the elements they belong to (no padded lane or k)."""
    g = np.random.default_rng(5)
    A, B = g.uniform(-1, 1, (45, 37)), g.uniform(-1, 1, (37, 29))
    A[3, :], B[:, 4] = -0.0, -0.0
    A[7, 36], B[36, 9], A[11, 2], B[5, 13] = np.inf, 0.0, np.nan, -np.inf
    D = torch.empty((29, 45), dtype=torch.float64, device="cuda").t()
    gbblas.jmul_(D, to_dev(A), to_dev(B))
    assert_bit_equal(to_host(D), oracle.jmul(np.asfortranarray(A), np.asfortranarray(B)))


@pytest.mark.parametrize("config", [0, 1, 2, 3, grouped.AUTO])
def test_grouped_edges_bit_exact(cuda, config):
    """Problems at the tile edges, empty ones, alpha = 0 and K = 0, first in the table and last."""
    sizes = [(0, 5, 4), (16, 16, 16), (17, 33, 31), (33, 17, 65), (64, 32, 33), (65, 64, 9), (63, 64, 12), (1, 200, 5),
             (130, 1, 40), (24, 24, 0), (40, 24, 8), (5, 0, 3)]
    alphas = [1.0, 1.0, 1.5, 1.0, 1.0, -1.0, 1.0, 1.0, 2.0, 1.5, 0.0, 1.0]
    betas = [0.0, 0.0, 0.5, 0.0, 1.0, 0.0, 0.0, 0.0, 0.25, 0.5, 0.5, 0.0]
    g = np.random.default_rng(11)
    h = [(g.uniform(-1, 1, (m, k)), g.uniform(-1, 1, (k, n)), g.uniform(-1, 1, (m, n))) for m, n, k in sizes]
    Cs = [to_dev(c) for _, _, c in h]
    plan = grouped.GroupedGemm([to_dev(a) for a, _, _ in h], [to_dev(b) for _, b, _ in h], Cs, alpha=alphas, beta=betas,
                               tuning=grouped.Tuning.from_list([config] * grouped.CLASSES))
    plan.run()
    first = [to_host(C) for C in Cs]
    for (a, b, c), C, al, be in zip(h, first, alphas, betas):
        if C.size:
            ref = oracle.gemm(np.asfortranarray(a), np.asfortranarray(b), C=np.asfortranarray(c), alpha=al, beta=be)
            assert_bit_equal(C, ref)
