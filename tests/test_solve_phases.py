"""The field solve's step is cut into phases by block barriers.  Thread 0 sets
the counters in shared memory back to zero; between that store and the next
use of the counter by another thread there must be a barrier, whichever way the
step ends (the window's barriers are only met when it moves).  Read from the
kernel's source: a step's phases are the stretches between the barriers that
every step meets.  The last stretch runs on into the next step's first, so a
counter that is reset there must not be counted up in either."""
from __future__ import annotations

import os
import re

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "fmt2d_b200", "csrc",
                   "eik64.cu")


def _step():
    """The step loop's body, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    start = text.index("for (; more; ++it) {")
    depth = 0
    for i in range(text.index("{", start), len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("no step loop")


def _phases():
    """Stretches of the step between the barriers at the loop's own depth; the
    batches of nodes at an interface end with a barrier each, so the loop over
    them ends a stretch as well (its body is the phase "evaluate")."""
    body = _step()
    out, cur, depth, i = [], "", 0, 0
    while i < len(body):
        if body.startswith("__syncthreads();", i) and depth == 1:
            out.append(cur)
            cur = ""
            i += len("__syncthreads();")
            continue
        if body.startswith("for (unsigned x0 = 0;;", i):
            d, j = 0, body.index("{", i)
            while True:
                d += {"{": 1, "}": -1}.get(body[j], 0)
                j += 1
                if d == 0:
                    break
            loop = body[i:j]
            assert loop.rstrip(" }\n").endswith("if (x0 + kXBatch >= nx) break;")
            assert loop.rindex("__syncthreads();") > loop.rindex("stage(")
            out.append(cur + loop)
            cur = ""
            i = j
            continue
        depth += {"{": 1, "}": -1}.get(body[i], 0)
        cur += body[i]
        i += 1
    # what follows the last barrier runs on into the next step's first stretch
    out[0] = cur + out[0]
    return out


def test_resets_and_uses_are_barriers_apart():
    ph = _phases()
    assert len(ph) == 3   # evaluate (with the end of the step before), arbitrate, spread
    evaluate, arbitrate, spread = ph
    # commits: counted in evaluate, read in arbitrate
    assert "place(&sh.nc" in evaluate and "nc = sh.nc;" in arbitrate
    assert not re.search(r"sh\.nc\s*=[^=]", evaluate)
    assert not re.search(r"sh\.nc\s*=[^=]", arbitrate)
    assert re.search(r"sh\.nc\s*=\s*0", spread) and "place(&sh.nc" not in spread
    # winners: counted in arbitrate, read in spread
    assert "place(&sh.nw" in arbitrate and "nw = sh.nw[0]" in spread
    assert re.search(r"sh\.nw\[0\]\s*=", evaluate)
    assert not re.search(r"sh\.nw\[0\]\s*=[^=]", arbitrate)
    assert not re.search(r"sh\.nw\[[01]\]\s*=[^=]", spread)
    # list lengths: read in evaluate, the read list's reset in arbitrate, which
    # with spread and the window lengthens the other list
    assert "sh.cnt[cur][0], nx = sh.cnt[cur][1]" in evaluate
    assert "sh.cnt[cur][0] = sh.cnt[cur][1] = 0u" in arbitrate
    assert not re.search(r"sh\.cnt\[cur\]\[[01]\]\s*=[^=]", evaluate + spread)
