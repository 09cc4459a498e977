"""Autotuning a size whose launches on CTA pairs cut tiles along K, and so have a band of their own: the
other bands are not candidates (they were timed as equals, and one of them installed by chance)."""
import pytest

from gbblas import tuning

pytestmark = pytest.mark.gpu


# M, N, K.  Cut on 76 pairs, by the costs of a cut (K panels of 64, three term products): 16 tiles of 128
# panels, 4 of 64, and for the adjoint 16 + 16 of 64 (two parts 3 * 32 * 64 / 76 + 32 = 113, whole
# 3 * 64 * 0.75 = 144; of 16 panels, at 1024^3, the parts would be 52 against 36, and nothing is cut).
@pytest.mark.parametrize("kind,shape", [("f32", (1024, 1024, 8192)), ("f32", (512, 300, 4096)), ("adjoint", (4096, 4096, 256))])
def test_one_band_on_pairs(cuda, kind, shape):
    for _ in range(3):
        t, ms = tuning.autotune(kind, *shape, reps=1, install=False)
        assert ms > 0 and (t.engine == 1 or t.band == 8)
