"""The ordered pair list at the edges of its search: groups of 32 leaves,
super-groups of 32 groups, candidate batches of 32, and each leaf width with a
form of its own (2 and 4 atoms, any other), bit for bit against the oracle's
rope walk."""
import numpy as np
import pytest

from helpers import uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("apl", [2, 3, 4, 8])
@pytest.mark.parametrize("leaves", [2, 31, 32, 33, 65, 1023, 1025, 2049])
def test_ordered_pairs_at_group_edges(nd, oracle, apl, leaves):
    n = apl * leaves
    x = uniform(1000 * apl + leaves, n)
    # a few pairs an atom, and a radius at which most leaves overlap
    for r in (np.float32(0.8 * n ** (-1.0 / 3.0)), np.float32(0.45)):
        if r > 0.4 and n > 4200:
            continue
        spec = nd.SpheresBVHSpecs(float(r), n, apl)
        for order in (0, 1):
            p = nd.leafbuild_traverse_bvh(x, spec, order=order)
            i, j, d = oracle.leaf_traverse(oracle.tree(x, float(r), apl, order=order), float(r), apl)
            assert len(p) == len(i)
            assert np.array_equal(p["i"], i) and np.array_equal(p["j"], j)
            assert np.array_equal(p["d"].view(np.int32), np.asarray(d, np.float32).view(np.int32))
