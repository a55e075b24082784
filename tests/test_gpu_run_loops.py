"""The run loops: steps are sent ahead of the host's looks at the control
block, and what the run is must not depend on how far."""
import ctypes as C

import pytest

from floodca_b200 import synth
from floodca_b200.lib import check, core, dropin
from floodca_b200.sim import DropinGrid, RunParams, Session
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _dom():
    return synth.config1(n=48, seed=5)[0]


@pytest.mark.parametrize("before", [0, 7])
def test_capped_run_that_reaches_its_time_sends_few_steps_more(before):
    """max_steps as a generous cap on a run that T_sim ends."""
    dom, p = _dom(), RunParams(steps=10**6, T_sim=600.0)
    want = pyoracle.run(dom, p.with_(steps=0))
    with Session(dom, p) as s:
        n0 = s.launches()
        s.advance(before)
        s.run()
        st = s.stats()
        assert st["step"] == want["step"] and st["t"] == want["t"]
        assert s.launches() - n0 < st["step"] + 256 + 2
        assert (s.download()[0] == want["h"]).all()


@pytest.mark.parametrize("before", [0, 33])
def test_fixed_count_sends_no_step_too_many(before):
    dom, p = _dom(), RunParams(steps=100, T_sim=1e6)
    with Session(dom, p) as s:
        n0 = s.launches()
        s.advance(before)
        s.run()
        assert s.stats()["step"] == 100
        assert s.launches() - n0 <= 100 + 1          # and the volume of the stats


def test_dropin_capped_run_equals_the_run_by_time():
    dom = _dom()
    a = DropinGrid(dom, RunParams(steps=10**6, T_sim=600.0))
    b = DropinGrid(dom, RunParams(T_sim=600.0))
    assert a.run() == 0 and b.run() == 0
    ra, rb = a.result(), b.result()
    assert ra["step"] == rb["step"] and (ra["h"] == rb["h"]).all()


@pytest.mark.parametrize("precision,nr,nc", [("f32", 260, 270), ("f64", 70, 65), ("f32", 40, 50)])
@pytest.mark.parametrize("expect", [-1, 0, 4095, 4096])
def test_steps_sent_with_and_without_a_graph(precision, nr, nc, expect):
    """Kernels with a device-side launch (FP32 above 2^16 cells, FP64) and
    without: sent one by one or as graphs, and changing over in the middle, the
    run is the same."""
    dom = synth.make_terrain(synth.TerrainSpec(nr, nc, seed=2))
    dom.h[:] = 0.02
    p = RunParams(steps=150, T_sim=1e6)
    want = pyoracle.run(dom, p, double=precision == "f64")
    with Session(dom, p, precision=precision) as s:
        check(core().fcab_sim_expect_steps(s.h, expect), "expect_steps")
        s.advance(70)
        check(core().fcab_sim_expect_steps(s.h, 10**6), "expect_steps")
        s.run()
        assert s.stats()["step"] == 150
        h = s.download()[0]
    if precision == "f32":
        assert (h == want["h"]).all()
    else:
        assert abs(h - want["h"]).max() <= 1e-12


@pytest.mark.parametrize("every", [1, 10, 37, 100])
@pytest.mark.parametrize("steps,T_sim", [(230, 1e6), (10**6, 600.0), (0, 600.0)])
def test_polled_runs_pause_where_they_should(every, steps, T_sim):
    """The ensemble session's poll hook in runs of a fixed count, a cap that
    the time undercuts, and a time: called at every multiple of poll_every
    short of the end, and the run is that of a session without pauses."""
    dom, p = _dom(), RunParams(steps=steps, T_sim=T_sim)
    L = dropin(False)
    plain = DropinGrid(dom, p)
    assert plain.run() == 0
    g = DropinGrid(dom, p)
    thr, fl, mx = (C.c_double * 1)(0.1), (C.c_long * 1)(), C.c_double()
    e = L.fca_cuda_ens_open(C.byref(g.g), C.byref(g.cfg), 1, thr)
    assert e
    calls = []
    hook = C.CFUNCTYPE(None, C.c_void_p)(lambda _: calls.append(1))
    try:
        assert L.fca_cuda_ens_run(e, C.byref(g.g), C.byref(g.cfg), C.byref(g.acc), C.byref(g.tm), fl,
                                  C.byref(mx), C.cast(hook, C.c_void_p), None, every) == 0
    finally:
        L.fca_cuda_ens_close(e)
    r = plain.result()
    assert g.acc.step == r["step"] and g.acc.t == r["t"]
    assert len(calls) == (r["step"] - 1) // every
    assert mx.value == float(r["hmax"].max())


@pytest.mark.parametrize("every", [7, 50])
def test_progress_lines_of_a_fixed_count(every, capfd):
    dom, p = _dom(), RunParams(steps=120, T_sim=1e6)
    want = pyoracle.run(dom, p)
    g = DropinGrid(dom, p)
    g.cfg.progress_every = every
    assert g.run() == 0
    r = g.result()
    assert r["step"] == 120 and (r["h"] == want["h"]).all()
    C.CDLL(None).fflush(None)
    lines = [ln for ln in capfd.readouterr().out.splitlines() if ln.startswith("progress step=")]
    assert [int(ln.split()[1].split("=")[1]) for ln in lines] == list(range(every, 120, every))
