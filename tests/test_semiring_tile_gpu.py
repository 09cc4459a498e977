"""The one-warp semiring tiles of float32 and int32 at their edges: 32 x 32 tiles, 16 k a panel, odd and
even K (k pairs), both operands in each orientation, leading dimensions that allow 8-byte copies and
ones that do not; and the large tiles that big outputs take.  Bit-identical to the oracle."""
import numpy as np
import pytest
import torch

import gbblas
import oracle
from gbblas import _lib
from gpu_util import assert_bit_equal, to_dev_ld, to_host

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 70, 17), (33, 1, 16), (32, 32, 15), (31, 33, 2), (65, 64, 31), (100, 90, 48), (500, 350, 33)]


def _operand(g, shape, dt):
    if dt == np.int32:
        return g.integers(-2 ** 31, 2 ** 31, shape).astype(np.int32)
    X = g.uniform(-2, 2, shape).astype(np.float32)
    X[g.uniform(size=shape) < 0.05] = np.nan
    X[g.uniform(size=shape) < 0.05] = -0.0
    X[g.uniform(size=shape) < 0.05] = np.inf
    return X


@pytest.mark.parametrize("dt", [np.float32, np.int32])
@pytest.mark.parametrize("sr", sorted(_lib.SEMIRINGS))
@pytest.mark.parametrize("pad", [0, 1])
def test_tile_edges_bit_exact(cuda, dt, sr, pad):
    g = np.random.default_rng(3 + pad)
    for M, N, K in SHAPES:
        for ta, tb, acc in ((0, 0, False), (1, 0, True), (0, 1, False), (1, 1, True)):
            A, B, C = _operand(g, (M, K), dt), _operand(g, (K, N), dt), _operand(g, (M, N), dt)
            ref = oracle.semiring_gemm(A, B, sr, C=C, accumulate=acc, dtype=dt)
            hold = lambda X, t: to_dev_ld(X.T if t else X, (X.shape[1 if t else 0] + 1) // 2 * 2 + pad, fill=3)  # noqa: E731
            Av, Bv = hold(A, ta)[0], hold(B, tb)[0]
            Cv, Cbuf = to_dev_ld(C, M + 1, fill=7)
            gbblas.gemm_semiring_(Cv, Av.t() if ta else Av, Bv.t() if tb else Bv, sr, accumulate=acc)
            assert_bit_equal(to_host(Cv), ref)
            assert np.all(to_host(Cbuf)[M:, :] == 7)


@pytest.mark.parametrize("dt", [np.float32, np.int32])
def test_large_output_bit_exact(cuda, dt):
    g = np.random.default_rng(9)
    A, B = _operand(g, (4096, 5), dt), _operand(g, (5, 4100), dt)
    Ad = torch.from_numpy(np.ascontiguousarray(A.T)).cuda().t()
    Bd = torch.from_numpy(np.ascontiguousarray(B.T)).cuda().t()
    C = to_host(gbblas.gemm_semiring(Ad, Bd, "min_plus"))
    rows = g.choice(4096, 40, replace=False)
    assert_bit_equal(np.asfortranarray(C[rows]), oracle.semiring_gemm(A[rows], B, "min_plus", dtype=dt))
