"""Rays share warps: several lanes step together, and a lane's step halvings
are tried by its neighbours.  A ray must come out the same, bit for bit,
whoever it shares a warp with: traced alone, in counts around a warp and a
block, and repeated until every warp is full; with and without rows."""
import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 31, 33, 65, 24000])
def test_ray_is_the_same_in_any_warp(count):
    from fmt2d_b200.api import Fmt2d
    phases = (1, 2, 3, 4, 5)
    m = synth.small_model(phases=phases, seed=11)
    g = Fmt2d(0).upload(m)
    g.forward(m.obs_x, phases)
    pk = m.picks
    src, ph = pk[:, 0].astype(np.int32), pk[:, 1].astype(np.int32)
    rx, rz = pk[:, 2], pk[:, 3]
    n = len(pk)
    t, valid, _ = g.trace(src, ph, rx, rz)
    rp, gi, gv = (a.copy() for a in g.frechet_rows(index_base=0))
    sel = np.random.default_rng(count).integers(0, n, count)
    t2, v2, _ = g.trace(src[sel], ph[sel], rx[sel], rz[sel])
    rp2, gi2, gv2 = g.frechet_rows(index_base=0)
    t3, v3 = g.trace_times(src[sel], ph[sel], rx[sel], rz[sel])
    assert t2.tobytes() == t[sel].tobytes() == t3.tobytes()
    assert np.array_equal(v2, valid[sel]) and np.array_equal(v3, valid[sel])
    for i in range(0, count, max(1, count // 200)):
        a, b = slice(rp2[i], rp2[i + 1]), slice(rp[sel[i]], rp[sel[i] + 1])
        assert np.array_equal(gi2[a], gi[b])
        assert gv2[a].tobytes() == gv[b].tobytes()
    g.close()
