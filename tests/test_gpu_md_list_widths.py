"""The list builds with leaves of 16 and 32 atoms, in blocks whose union is staged
and in blocks whose union is too large for it: the lists are exactly the pairs
within r_c + skin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(nd, oracle, x, side, apl):
    n, rl = len(x), 1.8
    p = nd.md_params(cutoff=1.5, skin=0.3, dt=1e-4, box_hi=(side,) * 3, atomsperleaf=apl,
                     rebuild_every=5)
    eng = nd.MDEngine(p, x, np.zeros((n, 3)))
    i, j, _ = eng.list_pairs()
    eng.close()
    ref = oracle.leaf_traverse(oracle.tree(x.astype(np.float32), rl, 2, order=1), rl, 2)
    a, b = np.asarray(ref[0], np.int64), np.asarray(ref[1], np.int64)
    want = np.sort(np.concatenate([a * (n + 1) + b, b * (n + 1) + a]))
    assert np.array_equal(np.sort(i.astype(np.int64) * (n + 1) + j), want)


@pytest.mark.parametrize("n,apl", [(8192, 8), (8192, 16), (8192, 32), (90112, 16), (90112, 32), (77840, 16),
                                   (77856, 32)])
def test_lists_of_unstaged_blocks(nd, oracle, n, apl):
    # a dense ball in a thin gas: its blocks' unions are far above the mean
    side = (n / 0.05) ** (1.0 / 3.0)
    rng = np.random.default_rng(n + apl)
    x = rng.uniform(0.0, side, (n, 3))
    k = 3000
    x[:k] = side / 2 + 3.2 * rng.uniform(-1.0, 1.0, (k, 3))
    _check(nd, oracle, rng.permutation(x), side, apl)
