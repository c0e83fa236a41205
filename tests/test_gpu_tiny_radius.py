"""Pair lists at radii whose square underflows in Float32: the lists still hold
every pair that the criterion accepts, between leaves as inside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [1e-30, 2e-23, 4e-23, 1e-22, 3e-20])
@pytest.mark.parametrize("mode", [0, 1])
def test_lists_where_the_square_underflows(nd, r, mode):
    # three leaves about the origin: coincident atoms, atoms a fraction of r apart
    x = np.zeros((12, 3), np.float32)
    x[4:, 0] = np.float32(0.37 * r)
    x[8:, 1] = np.float32(0.31 * r)
    spec = nd.SpheresBVHSpecs(r, 12, 4)
    with np.errstate(under="ignore"):
        d = x[:, None, :] - x[None, :, :]
        q = d * d
        d2 = (q[..., 0] + q[..., 1]) + q[..., 2]
        rf = np.float32(r)
        i, j = np.triu_indices(12, 1)
        for accept, call in ((np.sqrt(d2) < rf, nd.simdbuild_traverse_bvh),
                             (d2 < rf * rf, nd.leafbuild_traverse_bvh)):
            want = {(a + 1, b + 1) for a, b in zip(i, j) if accept[a, b]}
            p = call(x, spec, mode=mode, ctx=nd.Context())
            got = [(min(a, b), max(a, b)) for a, b in zip(p["i"].tolist(), p["j"].tolist())]
            assert len(got) == len(set(got)) and set(got) == want
