"""The functions that the block sweep evaluates on pairs, against correctly
rounded values: wherever one decides a rounding itself it has to be the right
one, and it may leave only a small share to the exact functions."""
import ctypes as C

import numpy as np
import pytest

from floodca_b200.lib import core

pytestmark = pytest.mark.gpu
G = np.float32(9.81)


def _probe(which, x, y=None, g=G):
    out = np.empty_like(x)
    vp = lambda a: None if a is None else a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert core().fcab_math_probe(which, vp(x), vp(y), vp(out), x.size, float(g)) == 0
    return out


def _depths(seed, n=3_000_000):
    rng = np.random.default_rng(seed)
    return np.concatenate([np.float32(2.0) ** rng.uniform(-20, 20, n).astype(np.float32),
                           np.linspace(1e-3, 10.0, n // 3, dtype=np.float32),
                           np.float32(2.0) ** np.arange(-20, 21).astype(np.float32)])


def test_cube_root_of_pairs():
    """Probe 10 with another value in the other half: the exact value (probe 0)
    or deferred, and deferred whenever either half cannot decide."""
    x = _depths(1)
    y = np.random.default_rng(2).permutation(x)
    exact, alone, pair = _probe(0, x), _probe(10, x), _probe(10, x, y)
    sure = ~np.isnan(alone)
    assert np.array_equal(alone[sure], exact[sure]) and sure.mean() > 0.995
    decided = ~np.isnan(pair)
    assert np.array_equal(pair[decided], exact[decided])
    assert np.array_equal(decided, sure & ~np.isnan(_probe(10, y)))
    assert (~sure).sum() > 100


def test_cube_root_defers_outside_its_range():
    x = np.float32([2.0 ** -21, 2.0 ** 21, 1e-30, 1e30, 3e38])
    assert np.isnan(_probe(10, x)).all()
    assert np.isnan(_probe(10, np.full_like(x, 0.5), x)).all()


@pytest.mark.parametrize("g", [9.81, 9.80665, 1.62, 3.0])
def test_critical_velocity_of_pairs(g):
    x = _depths(3)
    y = np.random.default_rng(4).permutation(x)
    g = np.float32(g)
    want = np.sqrt(np.float64(g) * x.astype(np.float64)).astype(np.float32)
    for got in (_probe(12, x, g=g), _probe(12, x, y, g=g)):
        decided = ~np.isnan(got)
        bad = np.flatnonzero(decided & (got != want))
        assert bad.size == 0, (x[bad[:5]], got[bad[:5]], want[bad[:5]])
        assert decided.mean() > 0.995


def test_root_of_the_slope():
    """Every float of two binades over a distance of 1 (both exponent parities
    of the square root), and random level differences over real distances."""
    mant = np.arange(0, 1 << 23, dtype=np.uint32)
    for e in (127, 128):
        x = ((np.uint32(e) << 23) | mant).view(np.float32)
        assert np.array_equal(_probe(13, x, g=1.0), np.sqrt(x))
    rng = np.random.default_rng(5)
    x = (10.0 ** rng.uniform(-5, 4, 4_000_000)).astype(np.float32)
    for d in (1.0, 10.0, 30.0, 90.0, np.float32(30.0 * 2 ** 0.5), 1e3):
        d = np.float32(d)
        assert np.array_equal(_probe(13, x, g=d), np.sqrt((x / d).astype(np.float32)))


def test_reciprocal_of_the_mean_manning_n():
    mant = np.arange(0, 1 << 23, dtype=np.uint32)
    for e in (120, 121):
        x = ((np.uint32(e) << 23) | mant).view(np.float32)
        assert np.array_equal(_probe(14, x), np.float32(1.0) / (np.float32(0.5) * x))
    x = np.float32([0.0, 1e-30, 1e-13, 2e-12, 3e-12, 1.0, 1e3])
    want = np.float32(1.0) / np.maximum(np.float32(0.5) * x, np.float32(1e-12))
    assert np.array_equal(_probe(14, x), want)


def test_unknown_probes_are_refused():
    x = np.ones(4, np.float32)
    vp = x.ctypes.data_as(C.c_void_p)
    for which in (-1, 15, 1, 6, 9, 11):
        assert core().fcab_math_probe(which, vp, None, vp, 4, 1.0) != 0
