"""Autotuning a size whose launches on CTA pairs cut tiles along K, and so have a band of their own: the
other bands are not candidates (they were timed as equals, and one of them installed by chance)."""
import pytest

from gbblas import tuning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [("f32", (1024, 1024, 8192)), ("f32", (512, 300, 4096)), ("adjoint", (1024, 1024, 1024))])
def test_one_band_on_pairs(cuda, kind, shape):
    for _ in range(3):
        t, ms = tuning.autotune(kind, *shape, reps=1, install=False)
        assert ms > 0 and (t.engine == 1 or t.band == 8)
