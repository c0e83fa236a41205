"""Engines of more than 4,096 blocks of 256 atoms, whose union search goes through
the boxes of super-blocks of 32 blocks: the same lists and steps, bit for bit, as
with the breadth-first tree search, refits inside the windows included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, seed):
    # a jittered lattice, loose enough for short lists
    k = int(np.ceil(n ** (1 / 3)))
    rng = np.random.default_rng(seed)
    at = np.stack(np.unravel_index(np.arange(n), (k, k, k)), axis=1).astype(np.float64)
    x = 1.5 * (at + 0.5) + rng.uniform(-0.2, 0.2, (n, 3))
    return x, rng.normal(0.0, 2.0, (n, 3)), 1.5 * k


# 4,097 blocks (a super-block of one), a ragged last block, 4,129 blocks
@pytest.mark.parametrize("n", [4096 * 256 + 4, 4128 * 256 + 128])
def test_two_level_search_equals_tree(nd, n):
    x, v, side = _state(n, n)
    res = []
    for search in (nd.ND_UNION_BLOCKS, nd.ND_UNION_TREE):
        mp = nd.md_params(cutoff=2.0, skin=0.2, dt=2e-3, box_hi=(side,) * 3, rebuild_every=8,
                          union_search=search)
        e = nd.MDEngine(mp, x, v, ctx=nd.Context())
        first = np.stack(e.list_pairs()[:2]).astype(np.int64)
        e.run(24)
        d = e.diagnostics()
        assert d["early_refits"] > 0 and d["skin_violations"] == 0
        last = np.stack(e.list_pairs()[:2]).astype(np.int64)
        res.append([np.sort(p[0] * (n + 1) + p[1]) for p in (first, last)] + list(e.get()))
        e.close()
    assert len(res[0][0]) > 10 * n
    for a, b in zip(*res):
        assert np.array_equal(a, b)
