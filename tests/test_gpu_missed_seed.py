"""Steps whose velocity maximum falls below the seed of the dt pruning: the
step has to take the full velocity pass before the next one. Up to 2^16 cells
the step's last CTA does it, beyond that a kernel launched from the step, in a
batch a second kernel: sizes on both sides of the line, with and without SEA
and WALL cells, K = 4 and 8, alone and as members of a batch.

The step rounds as the oracle does: depths are equal bit for bit, volumes are
sums of the same terms in another order (relative 1e-9)."""
import numpy as np
import pytest

from floodca_b200 import abi, synth
from floodca_b200.ensemble import Batch
from floodca_b200.sim import RunParams, Session, run_session
from oracle import pyoracle
from tests.test_gpu_block import _grid

pytestmark = pytest.mark.gpu
SIZES = [(256, 255), (256, 256), (256, 257), (300, 400)]


def _columns(nr, nc, masked):
    """Dry relief with a few one-cell water columns, which empty in about one
    step each."""
    dom = _grid(nr, nc, nr + nc, False)
    dom.h[:] = 0.0
    dom.Rday[:] = 0.0
    if masked:
        dom.mask[-3:, :] = abi.FCA_SEA
        dom.mask[:, :2] = abi.FCA_WALL
        dom.mask[nr // 2, nc // 3:nc // 2] = abi.FCA_WALL
        dom.mask[40:44, 60:64] = abi.FCA_SEA
    for r, c, depth in ((10, 10, 3.0), (45, 62, 2.0), (nr - 5, nc - 1, 1.6), (100, 56, 1.2), (150, 120, 0.7)):
        dom.h[r, c] = depth
    return dom


def _equal(got, want):
    assert got["step"] == want["step"] and got["t"] == want["t"]
    for k in ("h", "hmax", "tmax"):
        assert np.array_equal(got[k], want[k], equal_nan=True), k
    for k in ("V_bnd", "V_sea", "clamp_err"):
        assert got[k] == pytest.approx(want[k], rel=1e-9, abs=1e-9), k
    assert got["cap_active"] == want["cap_active"]


@pytest.mark.parametrize("K", [4, 8])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("size", SIZES)
def test_missed_seed(size, masked, K):
    dom = _columns(*size, masked)
    for p in (RunParams(K=K, steps=60, T_sim=1e6), RunParams(K=K, U=2, T_sim=700.0, edges=(1, 0, 0, 1))):
        want = pyoracle.run(dom, p)
        got = run_session(dom, p)
        assert got["dt_full_passes"] > 0
        _equal(got, want)


@pytest.mark.parametrize("K", [4, 8])
@pytest.mark.parametrize("masked", [False, True])
def test_missed_seed_in_a_batch(masked, K):
    p = RunParams(K=K, T_sim=700.0)
    doms = [_columns(nr, nc, masked) for nr, nc in SIZES]
    sessions = [Session(d, p) for d in doms]
    b = Batch(sessions)
    try:
        b.run(300.0)
        for d, s in zip(doms, sessions):
            st = s.stats()
            h, hmax, tmax = s.download()
            assert st["dt_full_passes"] > 0
            _equal({"h": h, "hmax": hmax, "tmax": tmax, **st}, pyoracle.run(d, p))
    finally:
        b.close()
        for s in sessions:
            s.close()


def _coast(n):
    d, p = synth.config1(n=n)
    d.mask[-4:, :] = abi.FCA_SEA
    d.mask[:, :1] = abi.FCA_WALL
    d.mask[n // 2, n // 3:n // 2] = abi.FCA_WALL
    return d, p


@pytest.mark.parametrize("n", [128, 300])
@pytest.mark.parametrize("K", [4, 8])
@pytest.mark.parametrize("masked", [False, True])
def test_fast_math_on_the_block_sweep(n, K, masked):
    """Hardware approximations against the exact run, within what fast math is
    held to: 1 mm of depth and 1e-5 of the volume."""
    d, p = _coast(n) if masked else synth.config1(n=n)
    p = p.with_(K=K)
    ex, fa = run_session(d, p), run_session(d, p, math="fast")
    land = d.mask == abi.FCA_LAND
    assert np.abs(ex["hmax"].astype(np.float64) - fa["hmax"])[land].max() <= 1e-3
    assert abs(ex["V"] - fa["V"]) <= 1e-5 * ex["V"]


@pytest.mark.parametrize("n", [128, 300])
@pytest.mark.parametrize("K", [4, 8])
def test_fp32_everywhere_on_masked_grids(n, K):
    """FP32 time and volumes on the block sweep: depths as on the row sweep in
    the same precision, bit for bit; volumes within float rounding."""
    d, p = _coast(n)
    p = p.with_(K=K, T_sim=1800.0)
    a = run_session(d, p, precision="f32all", cols_per_lane=1)
    b = run_session(d, p, precision="f32all")
    assert a["step"] == b["step"] and a["t"] == b["t"]
    for k in ("h", "hmax", "tmax"):
        assert np.array_equal(a[k], b[k]), k
    for k in ("V", "V_rain", "V_bnd", "V_sea"):
        assert b[k] == pytest.approx(a[k], rel=1e-4, abs=1e-3), k
