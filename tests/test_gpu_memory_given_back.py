"""Device memory of an engine goes back to the device when the caller destroys
it, and with it what the context kept of its forces() calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLACK = 8 << 20  # the driver's own granularity


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("make", ["engine", "ensemble", "adjoint"])
def test_closed_engine_gives_its_memory_back(nd, make):
    n, side = 65536, 45.0
    x = nd.synth.uniform_positions_mindist(3, n, side, 0.8)
    v = np.zeros((n, 3))
    ctx = nd.Context()
    mp = nd.md_params(skin=0.3, dt=1e-3, box_hi=(side,) * 3, rebuild_every=5)

    def used():
        if make == "adjoint":
            e = nd.Adjoint(mp, nd.adj_spec(25, checkpoint_every=25, bins=16), x, v, ctx=ctx)
            e.forward()
            e.backward()
            return e
        if make == "engine":
            e = nd.MDEngine(mp, x, v, ctx=ctx)
        else:
            table = nd.systems_table([n], [1.0], [1.0], [(0.0,) * 3], [(side,) * 3])
            e = nd.Ensemble(mp, table, x, v, ctx=ctx)
        e.run(5)
        e.get()
        return e

    nd.forces(x, None, nd.ForceField(), ctx=ctx)
    used().close()  # kernels loaded
    before = _free()
    e = used()
    assert before - _free() > 4 * SLACK
    e.close()
    assert _free() > before - SLACK
    # forces() keeps its buffers; closing any engine gives them back
    nd.forces(x, None, nd.ForceField(), ctx=ctx)
    assert before - _free() > 4 * SLACK
    used().close()
    assert _free() > before - SLACK


def test_list_pairs_beside_kept_buffers(nd):
    n, side = 4096, 17.0
    x = nd.synth.uniform_positions_mindist(3, n, side, 0.8)
    v = np.zeros((n, 3))
    mp = nd.md_params(skin=0.3, dt=1e-3, box_hi=(side,) * 3, rebuild_every=5)
    ctx, other = nd.Context(), nd.Context()
    nd.forces(x, None, nd.ForceField(), ctx=ctx)
    a, b = nd.MDEngine(mp, x, v, ctx=ctx), nd.MDEngine(mp, x, v, ctx=other)
    nd.forces(x, None, nd.ForceField(), ctx=ctx)
    for _ in range(2):
        rows = [np.stack(e.list_pairs()[:2]) for e in (a, b)]
        rows = [r[:, np.lexsort(r)] for r in rows]
        assert np.array_equal(*rows)
    a.close()
    b.close()
