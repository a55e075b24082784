"""The block sweep (FP32 grids) against the oracle, at the sizes
where its decomposition can go wrong: grids narrower than a strip, one column
past a strip, one row, rows one short of and one past a pass of eight, units
cut to one row, open edges at every side, an inflow cell on a strip's border,
and more strips than the GPU has CTAs.

The kernel rounds every operation as the oracle does, so FP32 results are
equal bit for bit; volumes are sums of the same terms in another order, with
float64 accumulation over at most 1e6 terms (relative 1e-9)."""
import numpy as np
import pytest

from floodca_b200.sim import Domain, RunParams, run_session
from oracle import pyoracle
from tests.test_oracle_random import _case

pytestmark = pytest.mark.gpu


def _grid(nr, nc, seed, rain_field, h0=0.03):
    rng = np.random.default_rng(seed)
    f = lambda a: a.astype(np.float32)  # noqa: E731
    z = 5.0 + 0.2 * np.arange(nr)[::-1, None] + rng.uniform(-1.5, 1.5, (nr, nc))
    rday = rng.uniform(0.0, 0.6, (nr, nc)) if rain_field else np.full((nr, nc), 0.4)
    return Domain(z=f(z), mask=np.zeros((nr, nc), np.uint8), n=f(rng.uniform(0.02, 0.15, (nr, nc))),
                  C=np.ones((nr, nc), np.float32), Rday=f(rday),
                  h=f(np.where(rng.random((nr, nc)) < 0.7, rng.uniform(0, h0, (nr, nc)), 0.0)),
                  dx=30.0)


def _check(dom, p, **kw):
    want = pyoracle.run(dom, p)
    got = run_session(dom, p, precision="f32", **kw)
    assert got["step"] == want["step"] and got["t"] == want["t"]
    for k in ("h", "hmax", "tmax"):
        assert np.array_equal(got[k], want[k], equal_nan=True), k
    for k in ("V_rain", "V_bnd", "V_sea", "clamp_err", "V_in"):
        assert got[k] == pytest.approx(want[k], rel=1e-9, abs=1e-9), k
    assert got["cap_active"] == want["cap_active"]
    assert got["cap_total"] == want["cap_total"]


SIZES = [(1, 1), (1, 200), (200, 1), (2, 56), (3, 57), (7, 112), (8, 113), (9, 55), (10, 64),
         (61, 93), (130, 59), (67, 300)]


@pytest.mark.parametrize("K", [4, 8])
@pytest.mark.parametrize("size", SIZES)
def test_block_sweep_sizes(size, K):
    nr, nc = size
    p = RunParams(K=K, steps=25, T_sim=1e6, hyeto="uniform", out_every=600.0, D_h=6.0)
    _check(_grid(nr, nc, 10 * nr + nc, False), p)
    _check(_grid(nr, nc, 7 * nr + nc, True), p.with_(hyeto="triangle", U=2))
    for edges in ((1, 0, 0, 0), (0, 0, 1, 0), (0, 1, 0, 1)):
        _check(_grid(nr, nc, 3 * nr + nc, False), p.with_(edges=edges))


@pytest.mark.parametrize("seg", [1, 2, 3, 10, 17])
def test_block_sweep_unit_heights(seg):
    """Units of every height, several to a CTA, an inflow cell beside a
    strip's border, deep water that reaches the critical velocity."""
    for nc, cell in ((113, 55), (120, 56), (300, 112)):
        p = RunParams(steps=20, T_sim=1e6, inflow_cell=5 * nc + cell, inflow_peak=400.0,
                      inflow_t_peak=600.0, inflow_t_end=1200.0)
        _check(_grid(70, nc, seg, seg % 2 == 0, h0=4.0), p, seg_rows=seg)


def test_block_sweep_more_strips_than_ctas():
    p = RunParams(steps=6, T_sim=1e6)
    _check(_grid(5, 36000, 4, True), p)
    _check(_grid(40, 36000, 5, False), p)


@pytest.mark.parametrize("seed", range(60))
def test_block_sweep_random(seed):
    dom, p = _case(5000 + seed)
    dom = dom.copy()
    dom.mask[:] = 0
    _check(dom, p)


def test_block_sweep_tiny_manning_and_dry_start():
    """Manning n of zero (clamped in the mean) and a dry start."""
    dom = _grid(33, 70, 3, False)
    dom.n[::3, ::2] = 0.0
    dom.n[1::3, 1::2] = 1e-13
    _check(dom, RunParams(steps=30, T_sim=1e6))
    dom.h[:] = 0.0
    _check(dom, RunParams(steps=30, T_sim=1e6, hyeto="uniform"))


@pytest.mark.parametrize("seed", range(60))
def test_block_sweep_random_masks(seed):
    """SEA and WALL cells anywhere, also under open edges."""
    dom, p = _case(7000 + seed)
    _check(dom, p)


@pytest.mark.parametrize("K", [4, 8])
@pytest.mark.parametrize("size", [(9, 55), (61, 93), (70, 113)])
@pytest.mark.parametrize("rain_field", [False, True])
def test_block_sweep_coast(size, K, rain_field):
    """A shore, wall blocks, and nodata (NaN, infinite, negative) in the
    rasters of cells that are not LAND, which the model never reads."""
    nr, nc = size
    dom = _grid(nr, nc, nr + nc, rain_field, h0=0.5)
    rng = np.random.default_rng(nc)
    rr, cc = np.mgrid[0:nr, 0:nc]
    dom.mask[(rr > 0.8 * nr + 2 * np.sin(0.3 * cc)) | (cc < 2)] = 1
    dom.mask[rng.random((nr, nc)) < 0.05] = 2
    off = dom.mask != 0
    dom.z[off] = rng.choice(np.float32([np.nan, np.inf, -9999.0, 3.0]), off.sum())
    dom.n[off] = rng.choice(np.float32([np.nan, 0.0, -1.0]), off.sum())
    dom.h[off] = rng.choice(np.float32([np.nan, np.inf, -9999.0, 0.0, 2.5]), off.sum())
    for z_sea in (0.0, 6.0):
        p = RunParams(K=K, steps=30, T_sim=1e6, out_every=600.0, z_sea=z_sea)
        _check(dom, p)
        _check(dom, p.with_(edges=(0, 1, 1, 0), hyeto="uniform"), seg_rows=3)
    _check(dom, RunParams(K=K, steps=12, T_sim=1e6, boundary="closed",
                          inflow_cell=int(np.flatnonzero(dom.mask.ravel() == 0)[5]),
                          inflow_peak=50.0, inflow_t_peak=100.0, inflow_t_end=900.0))


@pytest.mark.parametrize("K", [4, 8])
@pytest.mark.parametrize("zz", [-9e28, -1e30, -3.4028235e38, 3e29])
def test_block_sweep_coast_extreme_land_elevations(zz, K):
    """LAND cells with a raster's nodata as elevation, in rows with SEA and
    WALL cells and beside both: only the mask says which cells are SEA."""
    dom = _grid(40, 70, 3, False, h0=0.5)
    dom.mask[10:12, 20:24] = 1
    dom.mask[20, 30:40] = 2
    for r, c in ((11, 24), (12, 21), (11, 40), (20, 40), (20, 43), (30, 60)):
        dom.z[r, c] = np.float32(zz)
    _check(dom, RunParams(K=K, steps=20, T_sim=1e6, edges=(1, 0, 0, 0)))


SCALAR = [(1, 1, 0), (3, 27, 0), (16, 16, 0), (37, 53, 5), (130, 59, 0), (67, 300, 17), (511, 130, 0),
          (4, 63000, 0), (90, 31300, 0), (2600, 700, 0)]


@pytest.mark.parametrize("nr,nc,seg", SCALAR)
def test_row_sweep_ranges(nr, nc, seg):
    """The row sweep (one column to a lane; FP64's) at every way its rows are
    cut: ranges of one row, more strips than warps, an even split of long
    strips, cuts asked for. FP32 equals the oracle bit for bit; FP64 depths,
    each cell's own arithmetic, are the same however the rows are cut."""
    steps = 20 if nr * nc < 200000 else 4
    p = RunParams(steps=steps, T_sim=1e6, edges=(0, 1, 0, 1))
    _check(_grid(nr, nc, nr + nc, True), p, seg_rows=seg, cols_per_lane=1)
    dom = _grid(nr, nc, nr + 2 * nc, False)
    a = run_session(dom, p, precision="f64", seg_rows=seg)
    b = run_session(dom, p, precision="f64", seg_rows=nr)
    assert a["t"] == b["t"]
    for k in ("h", "hmax", "tmax"):
        assert np.array_equal(a[k], b[k], equal_nan=True), k
