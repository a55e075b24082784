"""A step whose row tile does not arrive within its bounded wait goes on with a
stale tile and leaves an error in the control block. Everything that reads the
run's state has to fail then, until the fields are uploaded again. The error is
put into the control block from the host; no transfer is lost."""
import ctypes as C

import numpy as np
import pytest

from floodca_b200 import synth
from floodca_b200.ensemble import Batch
from floodca_b200.lib import FcabError, check, core
from floodca_b200.sim import RunParams, Session
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _case():
    dom, _ = synth.config1(n=48, seed=3)
    return dom, RunParams(steps=20, T_sim=1e6)


def _lose_tile(s):
    check(core().fcab_sim_lost_tile_probe(s.h), "lost_tile_probe")


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_lost_tile_fails_every_reader_until_the_next_upload(precision):
    dom, p = _case()
    L = core()
    with Session(dom, p, precision=precision) as s:
        s.advance(10)
        assert s.poll().step == 10
        _lose_tile(s)
        for call in (s.poll, s.stats, s.download, s.count_flooded, s.run, s.stats):
            with pytest.raises(FcabError, match="row tile"):
                call()
        # a new clock does not make the depths good
        assert L.fcab_sim_reset_time(s.h, 0.0, 0, 0.0, -1) == 0
        with pytest.raises(FcabError, match="row tile"):
            s.download()
        d = s.dom
        assert L.fcab_sim_upload_state(s.h, d.h.ctypes.data_as(C.c_void_p), None, None) == 0
        assert L.fcab_sim_reset_time(s.h, 0.0, 0, 0.0, -1) == 0
        s.run()
        h = s.download()[0]
        assert s.stats()["step"] == 20
    if precision == "f32":
        assert np.array_equal(h, pyoracle.run(dom, p)["h"])


def test_lost_tile_fails_the_batch():
    dom, p = _case()
    sessions = [Session(dom, p) for _ in range(3)]
    b = Batch(sessions)
    try:
        _lose_tile(sessions[1])
        with pytest.raises(FcabError, match="member 1.*row tile"):
            b.run(0.0)
        assert sessions[0].stats()["step"] == 20
        with pytest.raises(FcabError, match="row tile"):
            sessions[1].download()
    finally:
        b.close()
        for s in sessions:
            s.close()
