"""Native FP32 products whose operands are packed first (copies with rows contiguous, padded to whole
tiles): either operand or both, k-contiguous and unaligned sources, ragged edges against the padded
remainder, alpha and beta, both ways round, kernel!.  The launches are counted, so that a test fails when
its shape is no longer packed: two of them eagerly, one under stream capture (no buffer in the graph).  All
bit-identical to the oracle's FMA chain."""
import numpy as np
import pytest
import torch

import gbblas
import oracle
from gpu_util import assert_bit_equal, to_dev, to_dev_ld, to_host

pytestmark = pytest.mark.gpu


def launches(call):
    before = gbblas.launch_counts().get("native_gemm", 0)
    call()
    torch.cuda.synchronize()
    return gbblas.launch_counts()["native_gemm"] - before


def ld_of(rows, pad):
    return (rows + 3) // 4 * 4 + pad


# (M, N, K), (transposed A, transposed B), leading dimensions beyond a multiple of 4 elements
CASES = [((1030, 1031, 1500), (1, 0), 3),    # both k-contiguous
         ((1030, 1031, 1500), (1, 0), 0),
         ((2111, 2050, 700), (1, 0), 1),     # larger tiles
         ((2111, 2050, 700), (0, 0), 0),     # B only
         ((2111, 2050, 700), (1, 1), 0),     # A only
         ((2050, 2111, 900), (0, 1), 1),     # unaligned rows, copied and not transposed
         ((3100, 45, 6001), (1, 0), 1),      # few columns, few rows
         ((45, 3100, 6001), (1, 0), 1)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%s-%d%d-%d" % (("x".join(map(str, c[0])),) + c[1] + (c[2],)))
@pytest.mark.parametrize("ab", [(1.0, 0.0), (1.5, 0.5)], ids=["jmul", "ab"])
def test_packed_bit_exact(cuda, case, ab):
    (M, N, K), (ta, tb), pad = case
    g = np.random.default_rng(M + N + K + pad)
    A, B, C = (np.asfortranarray(g.uniform(-1, 1, s).astype(np.float32))
               for s in ((K, M) if ta else (M, K), (N, K) if tb else (K, N), (M, N)))
    lds = [ld_of(X.shape[0], pad) for X in (A, B, C)]
    Av, _ = to_dev_ld(A, lds[0])   # NaN in the padding of A and B
    Bv, _ = to_dev_ld(B, lds[1])
    Cv, Cbuf = to_dev_ld(C, lds[2], fill=7.0)
    alpha, beta = ab
    n = launches(lambda: gbblas.gemm_raw(ta, tb, M, N, K, alpha, Av.data_ptr(), lds[0], Bv.data_ptr(), lds[1], beta,
                                         Cv.data_ptr(), lds[2], dtype=torch.float32,
                                         stream=torch.cuda.current_stream().cuda_stream))
    assert n == 2
    assert_bit_equal(to_host(Cv), oracle.gemm(A, B, C=C, alpha=alpha, beta=beta, trans_a=bool(ta), trans_b=bool(tb),
                                              dtype=np.float32))
    assert np.all(to_host(Cbuf)[M:, :] == 7.0)


def test_captured_call_takes_no_buffer_and_replays(cuda):
    M, N, K = 1030, 1031, 1500
    g = np.random.default_rng(8)
    A, B = (g.uniform(-1, 1, s).astype(np.float32) for s in ((M, K), (K, N)))
    Ad, Bd = torch.from_numpy(A).cuda(), to_dev(B)   # A row-major
    C = torch.empty((N, M), dtype=torch.float32, device="cuda").t()
    assert launches(lambda: gbblas.gemm_(C, Ad, Bd)) == 2
    first = to_host(C)
    assert_bit_equal(first, oracle.jmul(np.asfortranarray(A), np.asfortranarray(B), dtype=np.float32))
    C.zero_()
    graph = torch.cuda.CUDAGraph()

    def capture():
        with torch.cuda.graph(graph):
            gbblas.gemm_(C, Ad, Bd)

    torch.cuda.synchronize()
    assert launches(capture) == 1
    graph.replay()
    assert_bit_equal(to_host(C), first)


def test_kernel_packs_too(cuda):
    """kernel!'s X has k contiguous: D, read first, is the chain's start."""
    M, N, K = 2111, 2050, 700
    g = np.random.default_rng(9)
    D, A, X = (np.asfortranarray(g.uniform(-1, 1, s).astype(np.float32)) for s in ((M, N), (M, K), (K, N)))
    Dd = to_dev(D)
    assert launches(lambda: gbblas.kernel_(Dd, to_dev(A), to_dev(X))) == 2
    ref = oracle.kernel_chain(D.ravel(order="F"), A.ravel(order="F"), X.ravel(order="F"), M, N, M, K, K, dtype=np.float32)
    assert_bit_equal(to_host(Dd).ravel(order="F"), ref)
