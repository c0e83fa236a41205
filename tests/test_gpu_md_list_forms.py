"""The two list builds (a warp per leaf up to two blocks of 256 atoms per SM, a
thread per atom beyond) at every leaf width and ragged block ends: the engine's
lists are exactly the pairs within r_c + skin of the positions they were built
from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,apl", [(64, 1), (254, 2), (256, 4), (260, 4), (1288, 8), (1040, 16),
                                   (2080, 32), (38912, 4), (39168, 4), (39176, 8), (39200, 32),
                                   (77824, 4), (77832, 8)])
def test_lists_are_the_pairs_within_the_list_radius(nd, oracle, n, apl):
    side = (n / 0.83) ** (1.0 / 3.0)
    x, v, _ = nd.synth.lj_system(n, n, side, 0.8)
    rl = 1.8
    p = nd.md_params(cutoff=1.5, skin=0.3, dt=1e-4, box_hi=(side,) * 3, atomsperleaf=apl,
                     rebuild_every=5)
    eng = nd.MDEngine(p, x, 0.0 * v)
    i, j, near = eng.list_pairs()
    xf = x.astype(np.float32)
    eng.close()
    ref = oracle.leaf_traverse(oracle.tree(xf, rl, 4 if n % 4 == 0 else 2, order=1), rl,
                               4 if n % 4 == 0 else 2)
    a, b = np.asarray(ref[0], np.int64), np.asarray(ref[1], np.int64)
    want = np.sort(np.concatenate([a * (n + 1) + b, b * (n + 1) + a]))
    got = np.sort(i.astype(np.int64) * (n + 1) + j)
    assert np.array_equal(got, want)
    d = np.linalg.norm(xf[i - 1] - xf[j - 1], axis=1)
    assert np.array_equal(near.astype(bool) | (np.abs(d - 1.4) < 1e-5),
                          (d < 1.4) | (np.abs(d - 1.4) < 1e-5))
