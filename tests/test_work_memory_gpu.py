"""Workspaces of traces and gradients come from a memory pool that the engines of
a device share.  What it holds between calls must not be lost to the rest of
the process, must go with the last engine, and engines on several threads and
streams must not meet in it."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from fmt2d_b200 import synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _model(seed):
    return synth.small_model(nx=401, dx=0.25, zrel_max=21.5, nzs=87, n_obs=6, seed=seed)


def _args(m):
    pk = m.picks
    return (pk[:, 0].astype(np.int32), pk[:, 1].astype(np.int32), pk[:, 2].copy(), pk[:, 3].copy())


def _results(g, args):
    t, v, _ = g.trace(*args)
    rows = [a.copy() for a in g.frechet_rows(index_base=0)]
    r = g.misfit_gradient(*args, np.where(v, t + 0.01, -1.0), 0.04, want=("slow", "iface"))
    return [t, v, *rows, r["grad_slow"], r["grad_iface"]]


def _same(a, b):
    return all(x.tobytes() == y.tobytes() for x, y in zip(a, b))


def test_little_memory_leaves_nothing_behind():
    """With less than a quarter of the device to be had, a call frees what it took."""
    import torch
    from fmt2d_b200.api import Fmt2d
    m = _model(4)
    args = _args(m)
    g = Fmt2d(0).upload(m)
    g.forward(m.obs_x, (1, 3))
    free, total = torch.cuda.mem_get_info()
    fill = torch.empty(free - total // 5, dtype=torch.uint8, device="cuda")
    want = _results(g, args)
    before, _ = torch.cuda.mem_get_info()
    again = _results(g, args)
    after, _ = torch.cuda.mem_get_info()
    del fill
    torch.cuda.empty_cache()
    assert after == before
    assert _same(want, again) and _same(want, _results(g, args))
    g.close()


def test_engines_on_threads_share_the_pool():
    from fmt2d_b200.api import Fmt2d
    ms = [_model(5), _model(6), synth.small_model(seed=8)]
    gs = [Fmt2d(0).upload(m) for m in ms]
    for g, m in zip(gs, ms):
        g.forward(m.obs_x, (1, 3))
    want = [_results(g, _args(m)) for g, m in zip(gs, ms)]
    bad = []

    def work(k):
        try:
            for _ in range(5):
                if not _same(want[k], _results(gs[k], _args(ms[k]))):
                    bad.append(k)
        except Exception as e:   # noqa: BLE001 (reported below)
            bad.append((k, repr(e)))

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(gs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
    for g in gs:
        g.close()


def test_what_a_call_has_left():
    """In a process of its own: what the pool holds after a gradient PyTorch can
    have while the engines live, their next results are the same, and with the
    last engine the memory is free again."""
    code = """
import torch
from test_work_memory_gpu import MB, _args, _model, _results, _same
from fmt2d_b200.api import Fmt2d
m = _model(7)
free = lambda: torch.cuda.mem_get_info()[0]
def engine():
    g = Fmt2d(0).upload(m)
    g.forward(m.obs_x, (1, 3))
    return g
g = engine()                    # (the first calls load the library's code)
_results(g, _args(m))
g.close()
gs = [engine(), engine()]
f0 = free()
want = [_results(g, _args(m)) for g in gs]
f1 = free()
# six sources, three fields each, about 35,000 slots of some 300 bytes
assert f0 - f1 > 128 * MB, (f0, f1)
fill = torch.empty(f1 + 64 * MB, dtype=torch.uint8, device="cuda")
del fill
torch.cuda.empty_cache()
assert all(_same(w, _results(g, _args(m))) for w, g in zip(want, gs))
gs[0].close()
assert _same(want[1], _results(gs[1], _args(m)))
gs[1].close()
assert free() > f0, (f0, free())
"""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here]))
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)
