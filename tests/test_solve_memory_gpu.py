"""Device memory of a forward: per slot 73 bytes that stay with the field (time,
two gradients, seed, flags) and no more than 57 and two bits of scratch, so that
a batch of fields that filled the device still does."""
from __future__ import annotations

import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


def test_bytes_per_slot():
    import torch
    from fmt2d_b200.api import Fmt2d
    nsrc = 8
    m = synth.small_model(nx=4000, dx=0.1, zrel_max=52.0, nzs=105, n_obs=nsrc)
    small = synth.small_model(n_obs=1)
    g = Fmt2d(0).upload(small)
    g.forward(small.obs_x, (1,))     # (the library's code is loaded)
    g.upload(m)
    free0, _ = torch.cuda.mem_get_info()
    g.forward(m.obs_x, (1,))
    free1, _ = torch.cuda.mem_get_info()
    # rows from the highest seafloor node to the bottom, two interface rows
    rows = m.pgrid_nz() - int(np.floor(m.topo.min() / m.dx)) + 2
    slots = nsrc * rows * 4000
    # (an allocation takes up to 2 MB more: five a field, a dozen in all)
    assert free0 - free1 <= slots * (73 + 57.25) + (2 << 20) * (5 * nsrc + 12)
    g.close()
