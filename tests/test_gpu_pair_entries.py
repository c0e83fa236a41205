"""The pair list handed over as entries in one call, against the three-array
call on the same tree: same pairs, same order, same bits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _arrays(ctx, x, spec, order, simd=False):
    from naivedynamics import _lib
    from naivedynamics._lib import ptr
    from naivedynamics.bvh import _pairs
    f = _lib.lib().nd_simd_leaf_pairs if simd else _lib.lib().nd_leaf_pairs
    cs = spec.c_spec()
    return _pairs(lambda h, *a: f(h, ptr(x), ctypes.byref(cs), order, _lib.ND_PAIRS_ORDERED, *a), ctx)


# two leaves; ragged last block; generic leaf sizes; leaves of 16 (256 pairs a visit)
@pytest.mark.parametrize("n,apl,r", [(4, 2, 0.9), (8, 4, 0.0), (516, 4, 0.2), (1026, 2, 0.15),
                                     (999, 3, 0.2), (2048, 16, 0.25), (20004, 4, 0.06)])
@pytest.mark.parametrize("order", [0, 1])
def test_entries_match_arrays(nd, n, apl, r, order):
    rng = np.random.default_rng(n + apl)
    x = rng.random((n, 3), dtype=np.float32)
    ctx = nd.Context()
    spec = nd.SpheresBVHSpecs(r, n, apl)
    want = _arrays(ctx, x, spec, order)
    # a context without list memory, then one that has some, then one with enough
    for c in (nd.Context(), ctx, ctx):
        got = nd.leafbuild_traverse_bvh(x, spec, order=order, ctx=c)
        assert got.dtype == want.dtype and got.tobytes() == want.tobytes()
    if apl == 4:
        got = nd.simdbuild_traverse_bvh(x, spec, order=order, ctx=ctx)
        assert got.tobytes() == _arrays(ctx, x, spec, order, simd=True).tobytes()
    nl = nd.gpubvh_neighborlist(ctx, x, spec, order=order)
    assert nl.pairlist.tobytes() == want.tobytes()
    keys, pos, perm, _ = nd.leafTreeData(x, spec, order=order, ctx=ctx)
    k2, p2, perm2, _ = nl.treedata
    assert k2.tobytes() == keys.tobytes() and np.array_equal(perm2, perm)
    for a, b in zip(p2, pos):
        assert a.tobytes() == b.tobytes()


def test_list_memory_refused(nd):
    from naivedynamics import _lib
    from naivedynamics._lib import PAIR_DTYPE, ptr
    x = np.random.default_rng(1).random((64, 3), dtype=np.float32)
    spec = nd.SpheresBVHSpecs(0.5, 64, 4)
    cs = spec.c_spec()
    count = ctypes.c_int64()
    ctx = nd.Context()
    none = _lib.PAIR_ALLOC(lambda k, u: None)
    st = _lib.lib().nd_leaf_pair_list(ctx.handle, ptr(x), ctypes.byref(cs), 0, 0, None, None, None,
                                      0, None, None, None, None, none, None, ctypes.byref(count))
    assert st == _lib.ND_ERR_NOMEM
    fixed = np.empty(1, PAIR_DTYPE)
    fixed.flags.writeable = False
    nl = nd.gpubvh_neighborlist(ctx, x, spec)
    with pytest.raises(ValueError):
        nd.gpubvh_neighborlist_(fixed, nl.treedata, spec, ctx)
    again = nd.gpubvh_neighborlist_(nl.pairlist, nl.treedata, spec, ctx, position=x)
    assert again.pairlist.tobytes() == nd.leafbuild_traverse_bvh(x, spec, ctx=ctx).tobytes()
