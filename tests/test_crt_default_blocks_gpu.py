"""Blocks of a CRT call of a few tiles: one under the default tuning, however its values came to be
installed (reading and writing them back, an autotuner's run whose result is not installed), and the
panels of any other tuning."""
import pytest
import torch

import gbblas
from gbblas import tuning

pytestmark = pytest.mark.gpu

M, N, K = 2560, 1024, 64   # 40 tiles of 256 x 256, size class 1 (three panels by default)


@pytest.fixture
def blocks(cuda):
    A = torch.rand((K, M), dtype=torch.float64, device="cuda").t()
    B = torch.rand((N, K), dtype=torch.float64, device="cuda").t()
    C = torch.empty((N, M), dtype=torch.float64, device="cuda").t()

    def count():
        before = gbblas.launch_counts().get("ozaki_slice_mma", 0)
        gbblas.gemm_(C, A, B, mode="ozaki_crt", slices=12)
        torch.cuda.synchronize()
        return gbblas.launch_counts()["ozaki_slice_mma"] - before

    tuning.set_tuning("ozaki_crt", 1, None)
    yield count
    tuning.set_tuning("ozaki_crt", 1, None)


def test_default_tuning_read_and_written_back(blocks):
    assert tuning.size_class(M, N) == 1 and blocks() == 1
    tuning.set_tuning("ozaki_crt", 1, tuning.get_tuning("ozaki_crt", 1))
    assert blocks() == 1


def test_autotune_without_installing(blocks):
    assert blocks() == 1
    tuning.autotune("ozaki_crt", M, N, K, reps=1, install=False)
    assert blocks() == 1


def test_other_tunings_keep_their_panels(blocks):
    for panels, n in ((1, 1), (2, 2), (4, 4)):
        tuning.set_tuning("ozaki_crt", 1, {"engine": 2, "band": 8, "panels": panels})
        assert blocks() == n
    tuning.set_tuning("ozaki_crt", 1, {"engine": 2, "band": 4, "panels": 3})
    assert blocks() > 1
    tuning.set_tuning("ozaki_crt", 1, None)
    assert blocks() == 1
