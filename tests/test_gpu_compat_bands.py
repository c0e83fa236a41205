"""simulate! as written at the sizes where its Coulomb bands (256 rows, tiles of
four columns, one to several bands a block of the cluster) and its blocks of 32
Lennard-Jones rows begin and end: both Coulomb forms give the same bits, and
small sizes equal the oracle's literal loop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    a = np.array(a, np.float32, copy=True)
    a[np.isnan(a)] = np.nan
    return a.view(np.int32)


def _inputs(n, seed, side=1.0):
    rng = np.random.default_rng(seed)
    x = (side * rng.uniform(0.05, 0.95, (n, 3))).astype(np.float32)
    v = rng.normal(0.0, 1e-4, (n, 3)).astype(np.float32)
    m = rng.uniform(1.0, 5.0, n).astype(np.float32)
    q = rng.uniform(-1e-9, 1e-9, n).astype(np.float32)
    return x, v, m, q


def _run(nd, n, steps, side=1.0):
    x, v, m, q = _inputs(n, n, side)
    s = nd.GenericObjectCollection(x, v, mass=m, charge=q)
    clct = nd.GenericRandomCollector(objectnumber=n, minDim=(0.0,) * 3, maxDim=(side,) * 3,
                                     temperature=0.01)
    log = nd.simulate_compat_(s, nd.SimSpec(duration=steps, stepwidth=1, vDamp=0.0), clct)
    return np.asarray(log, np.float32), np.asarray(s.force, np.float32)


@pytest.mark.parametrize("n", [2, 5, 31, 33, 63, 65, 255, 256, 257, 513])
def test_bands_against_oracle(nd, oracle, n):
    x, v, m, q = _inputs(n, n)
    log, force = _run(nd, n, 2)
    ref = oracle.compat_simulate(x, v, np.zeros((n, 3)), m, q, (0.0,) * 3, (1.0,) * 3, 0.01, n, 1,
                                 2, 0.0)
    assert np.array_equal(_bits(log), _bits(ref[3]))
    assert np.array_equal(_bits(force), _bits(ref[2]))


@pytest.mark.parametrize("n,side", [(2047, 1.0), (2305, 2000.0), (4100, 0.01), (9000, 1.0)])
def test_bands_equal_levels(nd, monkeypatch, n, side):
    # side 2000 and 0.01: Lennard-Jones distances on both sides of the range
    # whose terms are Float32 pairs
    got = _run(nd, n, 2, side)
    monkeypatch.setenv("NAIVEGPU_COMPAT_GLOBAL", "1")
    want = _run(nd, n, 2, side)
    for a, b in zip(got, want):
        assert np.array_equal(_bits(a), _bits(b))
