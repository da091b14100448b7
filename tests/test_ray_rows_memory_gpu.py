"""Frechet rows are written into a pool while the rays are traced.  Where the
pool is too small for them (memory is short), the rays only count, and a
second trace writes: the rows are the same, bit for bit."""
import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,short", [(1, False), (3000, False), (24000, True)])
def test_rows_with_little_memory(count, short):
    import torch
    from fmt2d_b200._native import Fmt2dError
    from fmt2d_b200.api import Fmt2d
    phases = (1, 2, 3)
    m = synth.small_model(phases=phases, seed=5)
    pk = m.picks[np.arange(count) % len(m.picks)]
    args = (pk[:, 0].astype(np.int32), pk[:, 1].astype(np.int32), pk[:, 2].copy(), pk[:, 3].copy())

    def traced(leave):
        g = Fmt2d(0).upload(m)
        g.forward(m.obs_x, phases)
        fill = None
        if leave is not None:
            free, _ = torch.cuda.mem_get_info()
            fill = torch.empty(max(0, free - leave), dtype=torch.uint8, device="cuda")
        n0 = g.stats()["launches"]
        try:
            t, v, nnz = g.trace(*args)
            n = g.stats()["launches"] - n0
            r = [a.copy() for a in g.frechet_rows(index_base=0)]
        except Fmt2dError as e:
            assert "allocation" in str(e)
            return None
        finally:
            del fill
            torch.cuda.empty_cache()
            g.close()
        return t, v, nnz, r, n

    t, v, nnz, r, n = traced(None)
    assert nnz > 0
    # the pool takes up to a quarter of the free memory, the rows' assembly needs
    # the entries twice: the least memory that suffices, to a fifth, is too little
    # for the pool
    leave = 24 * nnz if short else None
    while (again := traced(leave)) is None:
        leave = leave * 6 // 5
    t2, v2, nnz2, r2, n2 = again
    assert n2 == n + (1 if short else 0)   # the second trace
    assert nnz2 == nnz and t.tobytes() == t2.tobytes() and np.array_equal(v, v2)
    assert all(a.tobytes() == b.tobytes() for a, b in zip(r, r2))


def test_kept_buffers_are_given_back():
    """What a trace with rows and a gradient keep for the next call goes back
    when another engine finds no memory, and both engines' results stay."""
    import torch
    from fmt2d_b200.api import Fmt2d
    m = synth.small_model(phases=(1, 3), seed=9)
    pk = m.picks[np.arange(6000) % len(m.picks)]
    args = (pk[:, 0].astype(np.int32), pk[:, 1].astype(np.int32), pk[:, 2].copy(), pk[:, 3].copy())

    def results(g):
        t, v, _ = g.trace(*args)
        rows = [a.copy() for a in g.frechet_rows(index_base=0)]
        grad = g.misfit_gradient(*args, np.where(v, t + 0.01, -1.0), 0.04, want=("slow",))
        return [t, v, *rows, grad["grad_slow"]]

    a = Fmt2d(0).upload(m)
    a.forward(m.obs_x, (1, 3))
    want = results(a)
    b = Fmt2d(0).upload(m)
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(max(0, free - (8 << 20)), dtype=torch.uint8, device="cuda")
    b.forward(m.obs_x, (1, 3))   # its fields do not fit beside what a has kept
    del fill
    torch.cuda.empty_cache()
    for g in (b, a):
        for x, y in zip(want, results(g)):
            assert x.tobytes() == y.tobytes()
        g.close()
