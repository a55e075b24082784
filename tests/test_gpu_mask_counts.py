"""The counts that an upload takes of its mask on the device: they decide which
sweep runs and what land_cells says, up to the 2^40 cells a session may have."""
import ctypes as C

import numpy as np
import pytest
import torch

from floodca_b200.lib import core

pytestmark = pytest.mark.gpu


def _counts(m, pitch, nr, nc):
    out = (C.c_longlong * 4)()
    assert core().fcab_mask_probe(C.c_void_p(m.data_ptr()), pitch, nr, nc, out) == 0
    return list(out)


@pytest.mark.parametrize("nr,nc", [(1, 1), (3, 130), (200, 77)])
def test_counts_of_a_mask(nr, nc):
    rng = np.random.default_rng(nr + nc)
    m = np.full((nr + 16, nc + 8), 2, np.uint8)
    m[8:8 + nr, 4:4 + nc] = rng.choice(np.uint8([0, 0, 0, 1, 2, 7]), (nr, nc))
    want = [int((m[8:8 + nr, 4:4 + nc] == v).sum()) for v in (0, 0, 1, 7)]
    assert _counts(torch.from_numpy(m).cuda(), nc + 8, nr, nc) == want


@pytest.mark.parametrize("value,at", [(0, 0), (1, 2), (9, 3)])
def test_counts_beyond_32_bits(value, at):
    """4100 rows of 2^20 cells, all of them one row in memory."""
    nr, nc = 4100, 1 << 20
    got = _counts(torch.full((nc + 8,), value, dtype=torch.uint8, device="cuda"), 0, nr, nc)
    assert nr * nc > 1 << 32
    assert got[at] == nr * nc
    assert got[1] == (nr * nc if value == 0 else 0)
