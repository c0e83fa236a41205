"""Adjoint engines of different sizes beside each other: a large one still runs
after a smaller one was made (the reverse kernel's shared memory limit belongs to
the process), with the gradients it has alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _make(nd, n, ctx):
    side = (n / 0.83) ** (1.0 / 3.0)
    x, v, _ = nd.synth.lj_system(0x4E440005, n, side, 0.8)
    mp = nd.md_params(cutoff=2.5, skin=0.3, dt=1e-3, box_hi=(side,) * 3, rebuild_every=5)
    return nd.Adjoint(mp, nd.adj_spec(25, checkpoint_every=25, bins=16), x, v, ctx=ctx)


def test_large_engine_after_a_smaller_one(nd):
    alone = _make(nd, 4096, nd.Context())
    want = alone.forward(), alone.backward()
    alone.close()
    large = _make(nd, 4096, nd.Context())
    small = _make(nd, 8, nd.Context())
    got = large.forward(), large.backward()
    small.forward()
    small.backward()
    assert got[0][0] == want[0][0] and np.array_equal(got[0][1], want[0][1])
    for k in want[1]:
        assert np.array_equal(got[1][k], want[1][k]), k
    large.close()
    small.close()
