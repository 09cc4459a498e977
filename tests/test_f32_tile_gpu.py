"""The packed-pair FP32 tiles: native and kernel! products at the edges of the tile shapes (16, 32 and
64 rows and columns, 16 k a panel), every orientation, aligned and unaligned leading dimensions, the
exchanged roles (few rows) and the packed operands (larger products; not under stream capture).
All bit-identical to the oracle's FMA chain."""
import numpy as np
import pytest
import torch

import gbblas
import oracle
from gpu_util import assert_bit_equal, to_dev, to_dev_ld, to_host

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 200, 17), (200, 1, 16), (3, 1000, 40), (31, 33, 15), (32, 16, 16), (33, 17, 33), (64, 64, 31),
          (65, 63, 48), (129, 130, 32), (520, 516, 36), (777, 1001, 45), (1030, 1284, 52)]


@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pad", [0, 3])
def test_native_edges_bit_exact(cuda, shape, trans, pad):
    """pad = 0 rounds the leading dimensions up to 16 bytes, pad = 3 leaves them unaligned."""
    M, N, K = shape
    ta, tb = trans
    g = np.random.default_rng(M * 31 + N * 17 + K + 2 * ta + tb)
    A = g.uniform(-1, 1, (K, M) if ta else (M, K)).astype(np.float32)
    B = g.uniform(-1, 1, (N, K) if tb else (K, N)).astype(np.float32)
    C = g.uniform(-1, 1, (M, N)).astype(np.float32)
    lds = [(X.shape[0] + 3) // 4 * 4 + pad for X in (A, B, C)]
    for alpha, beta in ((1.0, 0.0), (1.5, 0.5)):
        ref = oracle.gemm(np.asfortranarray(A), np.asfortranarray(B), C=np.asfortranarray(C), alpha=alpha, beta=beta,
                          trans_a=bool(ta), trans_b=bool(tb), dtype=np.float32)
        Av, _ = to_dev_ld(A, lds[0])   # NaN in the padding of A and B
        Bv, _ = to_dev_ld(B, lds[1])
        Cv, Cbuf = to_dev_ld(C, lds[2], fill=7.0)
        gbblas.gemm_raw(ta, tb, M, N, K, alpha, Av.data_ptr(), lds[0], Bv.data_ptr(), lds[1], beta, Cv.data_ptr(),
                        lds[2], dtype=torch.float32, stream=torch.cuda.current_stream().cuda_stream)
        assert_bit_equal(to_host(Cv), ref)
        assert np.all(to_host(Cbuf)[M:, :] == 7.0)


def test_captured_call_matches_and_replays(cuda):
    """Under stream capture no packing buffer is taken; the replay gives the same bits."""
    g = np.random.default_rng(8)
    A, B = (g.uniform(-1, 1, s).astype(np.float32) for s in ((900, 333), (333, 801)))
    Ad, Bd = to_dev(A), to_dev(B)
    C = torch.empty((801, 900), dtype=torch.float32, device="cuda").t()
    gbblas.gemm_(C, Ad, Bd)
    first = to_host(C)
    assert_bit_equal(first, oracle.jmul(np.asfortranarray(A), np.asfortranarray(B), dtype=np.float32))
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        gbblas.gemm_(C, Ad, Bd)
    C.zero_()
    graph.replay()
    assert_bit_equal(to_host(C), first)


@pytest.mark.parametrize("shape", [(1, 1, 5), (16, 40, 33), (33, 65, 17), (300, 290, 40)])
def test_kernel_edges_bit_exact(cuda, shape):
    M, N, K = shape
    g = np.random.default_rng(M + N + K)
    D, A, X = (g.uniform(-1, 1, s).astype(np.float32) for s in ((M, N), (M, K), (K, N)))
    Dd = to_dev(D)
    gbblas.kernel_(Dd, to_dev(A), to_dev(X))
    ref = oracle.kernel_chain(D.ravel(order="F"), A.ravel(order="F"), X.ravel(order="F"), M, N, M, K, K, dtype=np.float32)
    assert_bit_equal(to_host(Dd).ravel(order="F"), ref)


def test_special_values_stay_where_they_belong(cuda):
    """-0 chains, subnormals, Inf * 0 and NaN reach only their own rows and columns."""
    g = np.random.default_rng(5)
    A, B = (g.uniform(-1, 1, s).astype(np.float32) for s in ((45, 37), (37, 29)))
    A[3, :], B[:, 4] = -0.0, -0.0
    A[20, :] *= np.float32(1e-38)
    B[:, 21] *= np.float32(1e-5)
    A[7, 36], B[36, 9], A[11, 2], B[5, 13] = np.inf, 0.0, np.nan, -np.inf
    D = torch.empty((29, 45), dtype=torch.float32, device="cuda").t()
    gbblas.jmul_(D, to_dev(A), to_dev(B))
    assert_bit_equal(to_host(D), oracle.jmul(np.asfortranarray(A), np.asfortranarray(B), dtype=np.float32))
