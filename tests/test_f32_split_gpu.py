"""Term products and adjoints whose tiles are cut along K over several CTA pairs: one tile and a few of
them (every tile cut, parts of several lengths), outputs with a remainder after full rounds, unequal
contraction lengths in the two halves of an adjoint, beta, padded C.  The bound is the modes' own
(tolerance + K 2^-24) |A||B| (a sum in parts has no more roundings than one in a row), and two calls give
the same bits: the parts are summed in order, whoever comes last."""
import numpy as np
import pytest
import torch

import gbblas
from gpu_util import assert_bit_equal, to_dev, to_dev_ld, to_host

pytestmark = pytest.mark.gpu

TOL = {"bf16x3": 2.0 ** -15, "bf16x6": 2.0 ** -21}
# one tile; 2 x 1; 3 x 2 ragged; 12 x 10 = 120 tiles (a full round of 76 pairs and a remainder); 9 x 17 = 153
SHAPES = [(200, 130, 9000), (512, 200, 4100), (700, 300, 3001), (3001, 2503, 300), (2300, 4300, 321)]


@pytest.mark.parametrize("mode", ["bf16x3", "bf16x6"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_within_bound_and_deterministic(cuda, mode, shape, beta):
    M, N, K = shape
    g = np.random.default_rng(M + N + K)
    A, B = (g.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N)))
    C0 = g.standard_normal((M, N)).astype(np.float32)
    Ad, Bd = to_dev(A), to_dev(B)
    out = []
    for _ in range(2):
        Cv, buf = to_dev_ld(C0, M + 4, fill=7.0)
        gbblas.gemm_(Cv, Ad, Bd, 1.5, beta, mode=mode)
        torch.cuda.synchronize()
        gbblas.check_device_status()
        assert np.all(to_host(buf)[M:, :N] == 7.0)
        out.append(to_host(Cv))
    assert_bit_equal(out[0], out[1])
    rows = g.choice(M, min(M, 64), replace=False)
    A64, B64 = A[rows].astype(np.float64), B.astype(np.float64)
    ref = 1.5 * (A64 @ B64) + beta * C0[rows]
    absprod = 1.5 * (np.abs(A64) @ np.abs(B64))
    bound = (TOL[mode] + K * 2.0 ** -24) * absprod + 2.0 ** -22 * (np.abs(ref) + np.abs(beta * C0[rows]))
    err = np.abs(out[0][rows] - ref)
    assert np.all(err <= bound), float(np.max(err / bound))


@pytest.mark.parametrize("shape", [(300, 5000, 129), (5000, 260, 300), (1300, 700, 2100), (2600, 2300, 1030)])
def test_adjoint_within_bound_and_deterministic(cuda, shape):
    M, N, K = shape
    g = np.random.default_rng(M + N + K)
    A, B, W = (g.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (M, N)))
    got = []
    for _ in range(2):
        dA = torch.full((K, M), float("nan"), dtype=torch.float32, device="cuda").t()
        dB = torch.full((N, K), float("nan"), dtype=torch.float32, device="cuda").t()
        gbblas.gemm_adjoint_(dA, dB, to_dev(A), to_dev(B), to_dev(W))
        torch.cuda.synchronize()
        gbblas.check_device_status()
        got.append((to_host(dA), to_host(dB)))
    assert_bit_equal(got[0][0], got[1][0])
    assert_bit_equal(got[0][1], got[1][1])
    A64, B64, W64 = (x.astype(np.float64) for x in (A, B, W))
    for x, left, right, n in ((got[0][0], W64, B64.T, N), (got[0][1], A64.T, W64, M)):
        err = np.abs(x - left @ right)
        assert np.all(err <= (2.0 ** -15 + n * 2.0 ** -24) * (np.abs(left) @ np.abs(right)) + 1e-30)
