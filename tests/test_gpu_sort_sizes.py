"""The sort behind every list and rebuild at the edges of its three forms (one
block, one kernel a pass, counting and scanning kernels) and of their tiles:
codes and permutation equal a stable sort of the reference's codes."""
import numpy as np
import pytest

from helpers import uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 1020, 1024, 1028, 2048, 2052, 4096, 4100, 20000, 32768, 32772, 131072, 131076,
                               524288, 524292])
@pytest.mark.parametrize("same", [False, True])
def test_tree_order_is_a_stable_sort(nd, oracle, n, same):
    x = np.full((n, 3), 0.25, np.float32) if same else uniform(n, n)
    for order in (0, 1):
        _, pos, perm, _ = nd.leafTreeData(x, nd.SpheresBVHSpecs(0.01, n, 4), order=order)
        t = oracle.tree(x, 0.01, 4, order=order)
        assert np.array_equal(perm, t["perm"] + 1)
        assert np.array_equal(pos.morton_code, t["code"])


@pytest.mark.parametrize("n", [1, 31, 4096, 4097, 100000, 600000])
def test_sortperm(nd, n):
    import torch
    from naivedynamics import _lib
    rng = np.random.default_rng(n)
    # many equal keys among all 31 bits
    k = rng.integers(0, 2 ** 31, n, dtype=np.int64) & np.where(rng.random(n) < 0.5, 0x7F, 2 ** 31 - 1)
    k = k.astype(np.int32)
    kt = torch.from_numpy(k.copy()).cuda()
    perm = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx = nd.default_context()
    ctx.check(_lib.lib().nd_sortperm_dev(ctx.handle, kt.data_ptr(), n, perm.data_ptr()))
    want = np.argsort(k, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), want)
    assert np.array_equal(kt.cpu().numpy(), k[want])
