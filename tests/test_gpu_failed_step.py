"""A step that ends between two stages leaves nothing behind that a later call
reads: with CASL_CHECK=1 the library looks at the nodes after every stage, and a
stage that moves them out of the domain ends the step there, with the next
stage's crossings already counted.  The gridded PV of the state loaded next,
and the fields of the next run, are those of a handle that made no such step
(the same kernels on the same contours: equal to the last bit).

The variable is read once per process, so each case runs in its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import numpy as np
from hydra_b200.casl import CaslError, CaslGPU
from hydra_b200.synthetic import random_pv

n, beta = %d, %r
kw = dict(ncontq=20, beta=beta, dtmax=0.05, npm=1 << 18, nm=1 << 14)
g, f = CaslGPU(n, **kw), CaslGPU(n, **kw)
f.initialise(random_pv(n, 5.0, 8))
good = f.contours()
assert 0 < good["nptq"] <= 148 * 1024  # the stages count crossings
g.initialise(random_pv(n, 4.0, 7))
qs = g.field("qs")
qs[1, 1] = np.nan
g.set_field("qs", qs)
try:
    g.step(1)
except CaslError as e:
    assert e.code == 5, e.code
else:
    raise AssertionError("a step with a velocity that is not finite returned no error")
g.set_contours(good)
assert np.array_equal(g.con2grid(), f.con2grid())
q1 = random_pv(n, 6.0, 9)
for s in (g, f):
    s.initialise(q1)
for name in ("qs", "qc", "qd", "qspre"):
    assert np.array_equal(g.field(name), f.field(name)), name
for s in (g, f):
    s.step(2)
cg, cf = g.contours(), f.contours()
assert cg["nptq"] == cf["nptq"] and np.array_equal(cg["xq"], cf["xq"])
print("ok")
"""


@pytest.mark.parametrize("n,beta", [(32, 0.0), (64, 10.0), (128, 0.0)])
def test_state_after_a_failed_step(gpu_lib, n, beta):
    env = dict(os.environ, CASL_CHECK="1", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CODE % (n, beta)], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
