"""simulate! as written on both sides of the size from which its Coulomb part runs
in bands: equal to the oracle's literal loop, a rescaled step included."""
import numpy as np
import pytest

from test_gpu_compat_bands import _bits, _inputs, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 18])
def test_few_atoms_against_oracle(nd, oracle, n):
    x, v, m, q = _inputs(n, n)
    log, force = _run(nd, n, 11)
    ref = oracle.compat_simulate(x, v, np.zeros((n, 3)), m, q, (0.0,) * 3, (1.0,) * 3, 0.01, n, 1,
                                 11, 0.0)
    assert np.array_equal(_bits(log), _bits(ref[3]))
    assert np.array_equal(_bits(force), _bits(ref[2]))
