"""The FP64 semirings on element-dealt tiles and ordered integer keys, at the edges of both: tiles of 1 to
64 rows, panels of 8 to 32 k, each orientation, padded leading dimensions; NaNs of either sign,
infinities, both zeros, subnormals and the largest numbers.  (+) is exact, so bit-identical to the oracle."""
import numpy as np
import pytest

import gbblas
import oracle
from gbblas import _lib
from gpu_util import assert_bit_equal, to_dev_ld, to_host

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (3, 70, 17), (33, 1, 8), (16, 16, 33), (32, 33, 2), (65, 64, 31), (130, 257, 40), (500, 350, 65)]
SPECIAL = np.array([np.nan, -np.nan, np.inf, -np.inf, 0.0, -0.0, 5e-324, -5e-324, 1.7976931348623157e308,
                    -1.7976931348623157e308, 1.0, -1.0])


def _operand(g, shape, special):
    X = g.uniform(-2, 2, shape)
    hit = g.uniform(size=shape) < special
    X[hit] = g.choice(SPECIAL, int(hit.sum()))
    return X


@pytest.mark.parametrize("sr", sorted(_lib.SEMIRINGS))
@pytest.mark.parametrize("special", [0.1, 1.0])
def test_tile_edges_bit_exact(cuda, sr, special):
    g = np.random.default_rng(17)
    for M, N, K in SHAPES:
        for ta, tb, acc in ((0, 0, False), (1, 0, True), (0, 1, True), (1, 1, False)):
            A, B, C = (_operand(g, s, special) for s in ((M, K), (K, N), (M, N)))
            with np.errstate(all="ignore"):
                ref = oracle.semiring_gemm(A, B, sr, C=C, accumulate=acc, dtype=np.float64)
            Av = to_dev_ld(A.T if ta else A, (K if ta else M) + 1, fill=3)[0]
            Bv = to_dev_ld(B.T if tb else B, (N if tb else K) + 2, fill=3)[0]
            Cv, Cbuf = to_dev_ld(C, M + 1, fill=7)
            gbblas.gemm_semiring_(Cv, Av.t() if ta else Av, Bv.t() if tb else Bv, sr, accumulate=acc)
            assert_bit_equal(to_host(Cv), ref)
            assert np.all(to_host(Cbuf)[M:, :] == 7)


@pytest.mark.parametrize("sr", sorted(_lib.SEMIRINGS))
@pytest.mark.parametrize("nan", [np.nan, -np.nan])
def test_only_nan_products(cuda, sr, nan):
    """No number among the products: (+)'s identity, or C when accumulating."""
    A, B = np.full((20, 9), nan), np.full((9, 40), nan)
    C = np.full((20, 40), -3.0)
    for acc in (False, True):
        Cv = to_dev_ld(C, 20, fill=0)[0]
        gbblas.gemm_semiring_(Cv, to_dev_ld(A, 20, fill=0)[0], to_dev_ld(B, 9, fill=0)[0], sr, accumulate=acc)
        identity = np.inf if sr.startswith("min") else -np.inf
        assert_bit_equal(to_host(Cv), C if acc else np.asfortranarray(np.full((20, 40), identity)))
