"""A region with more rows than the solve block has words of shared memory for its
bitmap of moving nodes: rows that lie a power of two apart share a word, and the
step's stamp tells them apart.  50,000 rows of 12 columns, with and without a
time window: the fixed point of the one-thread stencil on every node, the same
bits for every block size, and the oracle's times."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle
from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [0.0, 64.0])
def test_more_rows_than_bitmap_words(window):
    from fmt2d_b200.api import Fmt2d
    m = synth.small_model(nx=12, dx=0.01, zrel_max=495.0, n_obs=1)
    assert m.pgrid_nz() > 50000
    x = float(m.obs_x[0])
    fields = None
    for threads in (384, 256):
        g = Fmt2d(0).upload(m).set_solve_threads(threads).set_full_check()
        g.set_schedule(window_cells=window)
        g.forward([x], (1,))
        f = g.field(0, 1)
        assert fields is None or all(a.tobytes() == b.tobytes() for a, b in zip(f, fields))
        fields = f
        g.close()
    o = pyoracle.Oracle(m)
    o.forward(0, x, 1)
    To, Tg = o.field(0, 1)[0], fields[0]
    both = (To < 1e19) & (Tg < 1e19)
    assert ((To < 1e19) != (Tg < 1e19)).sum() <= 2 and both.sum() > 400000
    assert np.abs(To[both] - Tg[both]).max() <= 5e-4
