"""Lists and engines of one context: what one call leaves in the context's
buffers must not reach another's results."""
import ctypes

import numpy as np
import pytest

from conftest import canon

pytestmark = pytest.mark.gpu


def _unordered(nd, x, spec, ctx):
    p = nd.leafbuild_traverse_bvh(x, spec, order=nd.ND_ORDER_SPATIAL, mode=nd.ND_PAIRS_UNORDERED,
                                  ctx=ctx)
    return canon(p["i"], p["j"], p["d"])


# The three list arrays get different sizes: entries grow the first alone, and
# blocks of dropped engines serve the others with more than was asked for.
# Every array has to bound what an unordered list writes.
@pytest.mark.parametrize("engines", [1, 3])
def test_unordered_lists_after_entries_and_engines(nd, engines):
    rng = np.random.default_rng(engines)
    side = 1000 ** (1 / 3) / 0.8 ** (1 / 3)
    xs, vs, _ = nd.synth.lj_system(7, 1000, side, 0.8)
    mp = nd.md_params(skin=0.3, dt=1e-3, box_hi=(side,) * 3, rebuild_every=5)
    ctx, other = nd.Context(), nd.Context()
    for _ in range(engines):
        nd.forces(xs, None, nd.ForceField(), ctx=ctx)
        nd.MDEngine(mp, xs, vs, ctx=ctx).close()
    pts = rng.random((512, 3), dtype=np.float32)
    spec = nd.SpheresBVHSpecs(0.2, 512, 4)
    entries = nd.leafbuild_traverse_bvh(pts, spec, ctx=ctx)
    assert len(entries) > 3000
    live = [nd.MDEngine(mp, xs, vs, ctx=c) for c in (ctx, other)]
    for r in (0.12, 0.2, 0.22, 0.25, 0.28, 0.31, 0.35):
        spec = nd.SpheresBVHSpecs(r, 512, 4)
        want = _unordered(nd, pts, spec, nd.Context())
        assert np.array_equal(_unordered(nd, pts, spec, ctx), want), r
        for e in live:
            e.run(5)
        for a, b in zip(live[0].get(), live[1].get()):
            assert np.array_equal(a, b), r
    for e in live:
        e.close()
