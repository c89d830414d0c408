"""Contour tracing (hydra_b200/csrc/trace.cuh) on fields that fill its tiles with
what smooth flows hold little of, against the oracle: noise (a saddle or a
small closed contour in most coarse cells), many levels per edge, a field
whose few contours cross whole tiles, and the grid open in y (beta != 0).

Bars: topology identical; nodes 1e-10, the bar of a recontouring from a field
alone."""
import numpy as np
import pytest

from hydra_b200.synthetic import random_pv

pytestmark = pytest.mark.gpu


def field(kind, n, seed):
    if kind == "noise":
        q = np.random.default_rng(seed).standard_normal((n, n))
        return q - q.mean()
    if kind == "wave":  # one mode: contours across the domain and back
        x = 2 * np.pi * np.arange(n) / n
        return np.sin(x)[:, None] + 0.5 * np.cos(x)[None, :] + 0.01
    return random_pv(n, n / 8.0, seed)


@pytest.mark.parametrize("kind,n,levels,beta", [
    ("noise", 32, 7, 0.0), ("noise", 32, 150, 0.0), ("noise", 64, 25, 0.0), ("noise", 32, 9, 10.0),
    ("noise", 64, 40, 10.0), ("wave", 32, 3, 0.0), ("wave", 128, 60, 0.0), ("wave", 64, 30, 10.0),
    ("flow", 32, 90, 0.0), ("flow", 64, 40, 0.0), ("flow", 64, 20, 10.0), ("flow", 256, 12, 0.0)])
def test_contours_of_a_field(oracle_mod, gpu_lib, kind, n, levels, beta):
    from hydra_b200.casl import CaslGPU
    q = field(kind, n, 3)
    kw = dict(ncontq=levels, beta=beta, dtmax=0.05, npm=1 << 20, nm=1 << 16)
    o, g = oracle_mod.Oracle(n, **kw), CaslGPU(n, **kw)
    o.initialise(q)
    g.initialise(q)
    co, cg = o.contours(), g.contours()
    assert (cg["nq"], cg["nptq"]) == (co["nq"], co["nptq"])
    for k in ("npq", "i1q", "i2q", "indq", "nextq"):
        assert np.array_equal(cg[k], co[k]), k
    for k in ("xq", "yq"):
        assert np.abs(cg[k] - co[k]).max() < 1e-10, k
    g.close()
    o.close()
