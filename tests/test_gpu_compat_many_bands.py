"""simulate! as written where a block of the Coulomb cluster runs six to ten
bands, whose terms go straight to registers: both Coulomb forms, same bits."""
import numpy as np
import pytest

from test_gpu_compat_bands import _bits, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [10241, 13313, 20477, 20480])
def test_many_bands_equal_levels(nd, monkeypatch, n):
    got = _run(nd, n, 2)
    monkeypatch.setenv("NAIVEGPU_COMPAT_GLOBAL", "1")
    want = _run(nd, n, 2)
    for a, b in zip(got, want):
        assert np.array_equal(_bits(a), _bits(b))
