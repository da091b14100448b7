"""The solver evaluates regular nodes with a form of the stencil that leaves out
the candidates it can tell to lose (reg_best), and the usual check after a solve
shares it.  Here the check evaluates every node with the one-thread stencil of
eik_eval.cuh, which forms all candidates, and compares time, gradient and flags
bit for bit: a forward raises when one node would change.  Models where the two
could differ: exact ties (one velocity everywhere), rough velocities, odd widths,
a source that coincides with an interface node, time windows, and fields so
large that the lists' bitsets do not fit in shared memory (one, then none)."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


def _model(kind, nx, dx, zrel, seed=0):
    m = synth.small_model(nx=nx, dx=dx, zrel_max=zrel, nzs=max(33, int(zrel / 0.5)), n_obs=1,
                          seed=seed + 7)
    rng = np.random.default_rng(seed)
    if kind == "even":
        return dataclasses.replace(m, vel=np.full_like(m.vel, 4.0))
    if kind == "rough":
        return dataclasses.replace(m, vel=rng.uniform(1.6, 8.0, m.vel.shape))
    if kind == "flat":     # flat interfaces on grid rows as well
        return dataclasses.replace(m, vel=np.full_like(m.vel, 4.0), topo=np.full(nx, 8 * dx),
                                   sed_z=np.full(nx, 16 * dx), moho_z=np.full(nx, 24 * dx))
    return m


CASES = [("model", 33, 0.25, 8.0, 0.0), ("model", 203, 0.25, 8.0, 8.0),
         ("even", 97, 0.25, 11.0, 0.0), ("even", 130, 0.2, 8.0, 4.0),
         ("rough", 65, 0.2, 8.0, 0.0), ("rough", 257, 0.25, 11.0, 16.0),
         ("flat", 120, 0.25, 8.0, 0.0), ("model", 1500, 0.25, 8.0, 0.0),
         ("model", 2001, 0.1, 33.0, 32.0), ("model", 4001, 0.1, 52.0, 32.0)]


@pytest.mark.parametrize("kind,nx,dx,zrel,window", CASES)
def test_every_node_by_the_whole_stencil(kind, nx, dx, zrel, window):
    from fmt2d_b200.api import Fmt2d, fields_of, phase_mask
    m = _model(kind, nx, dx, zrel)
    phases = (1, 2, 3, 4, 5) if nx < 1000 else (1, 3)
    tfs = fields_of(phase_mask(phases))
    # on a grid node; one whose depth is a seafloor node's where the grid has it
    x = 25.0 if (nx - 1) * dx > 30.0 else float(m.obs_x[0])
    want = None
    for full, threads in ((False, 384), (True, 384), (True, 256), (True, 512)):
        g = Fmt2d(0).upload(m).set_solve_threads(threads).set_full_check(full)
        g.set_schedule(window_cells=window)
        g.forward([x], phases)
        st = g.stats()
        assert st["unsettled"] == 0 and st["capped"] == 0
        got = [np.concatenate(g.field(0, tf)).tobytes() for tf in tfs]
        assert want is None or got == want
        want = got
        g.close()
