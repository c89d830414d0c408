"""The ranking of the contours' chains ends when nothing is left to change: with
contours of at most c chains, windows that grow fourfold a launch cover them all
after log4 c launches, and one more sees it.  CASL_TRACE=1 reports the launches
that did any work."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import numpy as np
from hydra_b200.casl import CaslGPU
n, kind = %d, %r
if kind == "noise":   # many small contours, and lists between saddles
    q = np.random.default_rng(3).standard_normal((n, n))
else:                 # cells of one wave: every contour about n/2 coarse cells long
    x = 2 * np.pi * np.arange(n) / n
    q = np.sin(3 * x + 0.3)[:, None] * np.sin(3 * x + 0.1)[None, :]
g = CaslGPU(n, ncontq=20, npm=1 << 20, nm=1 << 16)
g.initialise(q - q.mean())
print(g.counts()[0])
"""


@pytest.mark.parametrize("n,kind", [(64, "noise"), (128, "cells")])
def test_launches_that_do_work(gpu_lib, n, kind):
    env = dict(os.environ, CASL_TRACE="1", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CODE % (n, kind)], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    contours, chains = int(r.stdout), int(re.search(r"tracing: (\d+) chains", r.stderr)[1])
    a, b, rounds = map(int, re.search(r"ranking: (\d+) and (\d+) of (\d+) launches", r.stderr).groups())
    assert 4 ** (rounds - 1) >= chains > 4 ** (rounds - 2)
    # a coarse cell's contour piece crosses at most 32 fine lines, 2 of them
    # lines where chains end, and leaves by one: no contour here is longer
    # than a tenth of all chains
    assert contours >= 100
    assert a < rounds and b < rounds, (a, b, rounds, contours, chains)
