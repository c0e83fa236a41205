"""The unordered pair list at the edges of its search (groups of 32 leaves,
super-groups of 32 groups, a task list that has to grow) against the ordered
list of the same points: the same pairs, the same bits, each once."""
import numpy as np
import pytest

from helpers import uniform

pytestmark = pytest.mark.gpu


def _sorted(p):
    return np.sort(p, order=["i", "j", "d"]).tobytes()


@pytest.mark.parametrize("leaves", [2, 31, 32, 33, 64, 1023, 1025, 2049])
@pytest.mark.parametrize("shape", ["box", "clusters", "point"])
def test_unordered_matches_ordered(nd, leaves, shape):
    n = 4 * leaves
    x = uniform(77 + leaves, n)
    r = np.float32(0.9 * n ** (-1.0 / 3.0))
    if shape == "clusters":
        x[: n // 2] = 0.5 + 0.2 * (x[: n // 2] - 0.5)
    elif shape == "point":  # boxes of one size, some distances exactly zero
        if n > 256:
            pytest.skip("every pair is a hit")
        x[:] = x[0]
    spec = nd.SpheresBVHSpecs(float(r), n, 4)
    ctx = nd.Context()
    for order in (0, 1):
        a = nd.leafbuild_traverse_bvh(x, spec, order=order, mode=nd.ND_PAIRS_UNORDERED, ctx=ctx)
        b = nd.leafbuild_traverse_bvh(x, spec, order=order, ctx=ctx)
        assert _sorted(a) == _sorted(b)


def test_task_list_grows(nd):
    # in the reference order every group of leaves overlaps most others
    n = 65536
    x = uniform(5, n)
    spec = nd.SpheresBVHSpecs(0.008, n, 4)
    ctx = nd.Context()
    a = nd.leafbuild_traverse_bvh(x, spec, order=0, mode=nd.ND_PAIRS_UNORDERED, ctx=ctx)
    b = nd.leafbuild_traverse_bvh(x, spec, order=0, ctx=ctx)
    assert _sorted(a) == _sorted(b)
