"""Pair lists over more than 262,144 leaves, whose search has two levels more:
the pairs of the per-atom walk, in the order the reference emits them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# just below and above the line; a ragged end; a second node on the top level
@pytest.mark.parametrize("leaves,apl", [(262144, 2), (262145, 2), (262144 + 33, 4), (266241, 3),
                                        (2**20 + 32 * 32 + 1, 2)])
def test_order_and_pairs(nd, leaves, apl):
    check_list(nd, leaves, apl, 1.1)


def check_list(nd, leaves, apl, r):
    """The device list of leaves * apl points at density 0.52; its length."""
    import torch
    n, side = leaves * apl, 100.0 * (leaves * apl / 524288) ** (1 / 3)
    x = nd.synth.uniform_positions(leaves, n, side)
    spec = nd.SpheresBVHSpecs(r, n, apl)
    ctx = nd.Context()
    dev = torch.device("cuda")
    xd = torch.from_numpy(x).to(dev)
    cap = int((2 * r**3 + 1) * n)
    out = [torch.empty(cap, dtype=t, device=dev) for t in (torch.int32, torch.int32, torch.float32)]

    def listed(mode):
        torch.cuda.synchronize()
        st, k = nd.neighbor_pairs_dev(xd, spec, *out, cap, order=nd.ND_ORDER_SPATIAL, mode=mode,
                                      ctx=ctx)
        assert st == 0 and k > 0
        return k, nd.pair_hash_dev(*out, k, ctx=ctx)

    k, h = listed(nd.ND_PAIRS_ORDERED)
    first = {f: o[:k].cpu().numpy() for f, o in zip(("i", "j", "d"), out)}
    # query leaf, target leaf, atom of the one, atom of the other, each outer to
    # the next: increasing from entry to entry
    _, pos, _, _ = nd.leafTreeData(x, spec, order=nd.ND_ORDER_SPATIAL, ctx=ctx)
    slot = torch.empty(n + 1, dtype=torch.int64, device=dev)
    slot[torch.from_numpy(pos.index.astype(np.int64)).to(dev)] = torch.arange(n, device=dev)
    a, b = slot[out[0][:k].long()], slot[out[1][:k].long()]
    q, t = a // apl, b // apl
    outer = q * (leaves + 1) + t
    inner = (a % apl) * apl + b % apl
    assert bool((t >= q).all()) and bool((a < b).all())
    step = outer[1:] - outer[:-1]
    assert bool(((step > 0) | ((step == 0) & (inner[1:] > inner[:-1]))).all())
    if apl == 4:
        assert listed(nd.ND_PAIRS_UNORDERED) == (k, h)
    p = nd.build_traverse_bvh(x, spec, order=nd.ND_ORDER_SPATIAL, ctx=ctx, capacity_hint=k)
    assert len(p) == k
    w = [torch.from_numpy(np.ascontiguousarray(p[f])).to(dev) for f in ("i", "j", "d")]
    torch.cuda.synchronize()
    assert nd.pair_hash_dev(*w, k, ctx=ctx) == h
    entries = nd.leafbuild_traverse_bvh(x, spec, order=nd.ND_ORDER_SPATIAL, ctx=ctx)
    for f in first:
        assert np.array_equal(np.ascontiguousarray(entries[f]), first[f])
    return k
