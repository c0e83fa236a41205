"""A neighbour list that cannot be resized is refused with nothing changed: not
the list, not the tree data."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _readonly(a):
    a.flags.writeable = False
    return a


@pytest.mark.parametrize("form", ["read-only", "view", "strided"])
def test_refused_list_changes_nothing(nd, form):
    n = 516
    x = np.random.default_rng(1).random((n, 3), dtype=np.float32)
    spec = nd.SpheresBVHSpecs(0.2, n, 4)
    ctx = nd.Context()
    nl = nd.gpubvh_neighborlist(ctx, x, spec)
    base = np.ones(8, nd.PAIR_DTYPE)
    given = {"read-only": _readonly(base), "view": base[:4], "strided": base[::2]}[form]
    tree, pos, perm, _ = nl.treedata
    kept = [a.tobytes() for a in (base, tree, *pos, perm)]
    moved = x + np.float32(0.01)
    with pytest.raises(ValueError):
        nd.gpubvh_neighborlist_(given, nl.treedata, spec, ctx, position=moved)
    assert len(base) == 8 and [a.tobytes() for a in (base, tree, *pos, perm)] == kept
    again = nd.gpubvh_neighborlist_(nl.pairlist, nl.treedata, spec, ctx, position=moved)
    assert again.treedata[0].tobytes() != kept[1] and len(again.pairlist) > 0
