"""One host thread per context: the first calls of several contexts at once, in
a process that has launched nothing yet, give the reference walk's hits
(tolerance zero)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = r"""
import threading
import numpy as np
from aviatorengine2_b200 import Context, _lib, scenes
s = scenes.cornell_box(width=64, height=48)
rng = np.random.default_rng(1)
n = 60_000
rays = np.zeros(n, _lib.RAY)
o, d = rng.uniform(1, 9, (n, 3)), rng.normal(size=(n, 3))
for k, x in enumerate("xyz"):
    rays["o" + x], rays["d" + x] = o[:, k], d[:, k]
rays["tnear"] = 0.001
ctxs = [Context(64, 48) for _ in range(8)]
for c in ctxs:
    c.upload(s)
gate, got = threading.Barrier(len(ctxs)), [None] * len(ctxs)
def first(k):
    gate.wait()
    got[k] = ctxs[k].closest_hit(rays, _lib.VARIANT_FAST_WALK if k % 4 else _lib.VARIANT_FAST)
ts = [threading.Thread(target=first, args=(k,)) for k in range(len(ctxs))]
[t.start() for t in ts]
[t.join() for t in ts]
want = ctxs[0].closest_hit(rays, _lib.VARIANT_PLAIN).view(np.uint8)
assert all(np.array_equal(g.view(np.uint8), want) for g in got)
[c.close() for c in ctxs]
print("equal")
"""


@pytest.mark.parametrize("again", range(3))
def test_first_calls_of_several_contexts(again):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "equal" in r.stdout, r.stderr[-2000:]
