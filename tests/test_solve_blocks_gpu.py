"""Field solve over the sizes where its lists, bitmaps and lanes have edges:
grids of odd widths, a grid wide enough that the interface-seeded stages start
with more nodes than the shared-memory lists hold and wider than the moving
bitmap's 256 columns, a source on a grid node that coincides with an interface
node (the fixed node), and every block size.  The result must be the fixed
point of the one-thread stencil (the check of every node after the solve, which
evaluates it with eik_eval.cuh's functions and compares bit for bit, finds
nothing to change), the same bits for every block size and call, and reach the
nodes the oracle reaches."""
from __future__ import annotations

import numpy as np
import pytest

import pyoracle
from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu

SIZES = [(33, 0.25, 8.0), (65, 0.2, 8.0), (97, 0.25, 11.0), (203, 0.25, 8.0), (1500, 0.25, 8.0)]


@pytest.mark.parametrize("nx,dx,zrel", SIZES)
def test_block_sizes(nx, dx, zrel):
    from fmt2d_b200.api import Fmt2d, fields_of, phase_mask
    m = synth.small_model(nx=nx, dx=dx, zrel_max=zrel, nzs=33, n_obs=1)
    # a seafloor node of depth 3.0 km on a grid row when the grid reaches x = 25 km
    x = 25.0 if (nx - 1) * dx > 30.0 else float(m.obs_x[0])
    phases = (1, 2, 3, 4, 5) if nx < 1000 else (1, 3)
    tfs = fields_of(phase_mask(phases))
    fields = {}
    for threads in (256, 384, 512, 384):
        g = Fmt2d(0).upload(m).set_solve_threads(threads)
        g.forward([x], phases)      # raises when the check finds a node to change
        st = g.stats()
        assert st["unsettled"] == 0 and st["capped"] == 0
        for tf in tfs:
            f = np.concatenate(g.field(0, tf))
            if tf in fields:
                assert f.tobytes() == fields[tf].tobytes(), (threads, tf)
            fields[tf] = f
        g.close()
    o = pyoracle.Oracle(m)
    o.forward(0, x, phase_mask(phases))
    for tf in tfs:
        To = o.field(0, tf)[0]
        assert ((To < 1e19) != (fields[tf][:To.size] < 1e19)).sum() <= 2, tf
