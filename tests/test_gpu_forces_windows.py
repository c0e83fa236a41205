"""nd_forces takes no step: its window length changes neither its result nor the
memory it needs; and windows whose steps are checked sparsely keep a vote for each
checked step."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [-1, 0, 10, 2**31 - 9, 2**31 - 8, 2**31 - 1])
def test_forces_with_any_window(nd, every):
    from naivedynamics import _lib
    from naivedynamics._lib import ptr
    x, _, q = nd.synth.lj_system(5, 1000, 10.7, 0.8, charges=True)

    def forces(k):
        p = nd.md_params(coulomb_k=1.0, skin=0.0, box_hi=(10.7,) * 3, rebuild_every=k)
        f = np.empty((1000, 3), np.float32)
        e = ctypes.c_double()
        ctx = nd.Context()
        ctx.check(_lib.lib().nd_forces(ctx.handle, ctypes.byref(p), 1000, ptr(x), ptr(q), ptr(f),
                                       ctypes.byref(e)), "nd_forces")
        return f, e.value

    want, got = forces(1), forces(every)
    assert got[0].tobytes() == want[0].tobytes()
    # the energy's blocks are added in any order: at most 1,000 double additions of
    # terms whose sizes sum to less than ten times the energy
    assert abs(got[1] - want[1]) <= 1000 * 2.0**-53 * 10 * abs(want[1])


@pytest.mark.parametrize("every,check", [(1, 1), (2, 1), (2, 3), (7, 2), (8, 2), (9, 4), (10, 9)])
def test_checked_steps_vote(nd, every, check):
    # fast atoms, a thin skin: refits inside the windows; captured windows and
    # windows run step by step take the same ones
    side = 17.0
    x, v, _ = nd.synth.lj_system(9, 4096, side, 0.8)
    mp = nd.md_params(skin=0.2, dt=2e-3, box_hi=(side,) * 3, rebuild_every=every,
                      refit_check_every=check)
    a, b = nd.MDEngine(mp, x, v, ctx=nd.Context()), nd.MDEngine(mp, x, v, ctx=nd.Context())
    a.run(6 * every)
    for _ in range(6 * every):
        b.run(1)
    for p, q in zip(a.get(), b.get()):
        assert np.array_equal(p, q)
    da, db = a.diagnostics(), b.diagnostics()
    assert da["early_refits"] == db["early_refits"]
    if every >= 7 and check <= 2:
        assert da["early_refits"] > 0
    a.close()
    b.close()
