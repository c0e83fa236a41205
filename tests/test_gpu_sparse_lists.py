"""Ordered lists of many leaves, sparse (rope walks) and dense (wide search) on both
sides of the lines between them: the pairs of the per-atom walk, in the order the
reference emits them, as arrays and as entries; and over a kept order."""
import numpy as np
import pytest

from conftest import canon
from test_gpu_deep_search import check_list

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves,apl,r", [(131072, 4, 0.2), (131073, 4, 0.2), (131073, 4, 2.0),
                                          (131073, 2, 0.3), (131101, 3, 0.3), (262145, 3, 1.4),
                                          (262144, 8, 0.1), (2**20 + 1057, 2, 0.4),
                                          (2**20 + 1, 2, 2.0)])
def test_order_and_pairs(nd, leaves, apl, r):
    check_list(nd, leaves, apl, r)


# clusters: some leaves span two of them and are searched for among walks
@pytest.mark.parametrize("r,clusters", [(0.3, 0), (2.0, 0), (0.1, 8), (0.05, 64)])
def test_kept_order_and_tree(nd, r, clusters):
    n = 4 * 131136
    x = (nd.synth.cluster_positions(3, n, clusters, 400.0, 10.0, 40.0) if clusters
         else nd.synth.uniform_positions(5, n, 100.0))
    spec = nd.SpheresBVHSpecs(r, n, 4)
    ctx = nd.Context()
    nl = nd.gpubvh_neighborlist(ctx, x, spec, order=nd.ND_ORDER_SPATIAL)
    want = nd.leafbuild_traverse_bvh(x, spec, order=nd.ND_ORDER_SPATIAL, ctx=nd.Context())
    assert nl.pairlist.tobytes() == want.tobytes()
    keys = nd.leafTreeData(x, spec, order=nd.ND_ORDER_SPATIAL, ctx=ctx)[0]
    assert nl.treedata[0].tobytes() == keys.tobytes()
    again = nd.gpubvh_neighborlist_(None, nl.treedata, spec, ctx, position=x)
    assert again.pairlist.tobytes() == want.tobytes()
    assert np.array_equal(again.treedata[1].position, nl.treedata[1].position)
    by_atom = nd.build_traverse_bvh(x, spec, order=nd.ND_ORDER_SPATIAL, ctx=ctx,
                                    capacity_hint=len(want))
    assert np.array_equal(canon(*(by_atom[f] for f in "ijd")), canon(*(want[f] for f in "ijd")))
