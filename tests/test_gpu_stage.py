"""The four launches of an RK4 stage (hydra_b200/csrc/stage.cuh) at every grid
size they are instantiated for, against the oracle: one advance from a state
made by hand (an ellipse of nodes, spectral fields of random phases), so that
the sizes the oracle could not initialise are reached too.

Bars: those of the one-step parity tests, 1e-12 of the largest position and
velocity and 1e-11 of the largest spectral coefficient (rounding of an
n-point transform is a few eps log2 n, about 1e-14).  In the FP32-inversion
mode the velocity and the gradients are rounded to 2^-24 = 6e-8 of their
size; a position moves by dt |u| < 1, a field by dt times the products, so
1e-6 covers both with the sums over a stage."""
import numpy as np
import pytest

from hydra_b200.synthetic import ptospc_np, random_pv

pytestmark = pytest.mark.gpu

NONE, FULL = {}, dict(kd=2.5, beta=10.0, rekman=0.1, rtherm=0.05)


def ellipse(n, count):
    a = 2 * np.pi * np.arange(count) / count
    # across the periodic edge in x, so that wrapped segments are met
    x = (3.0 + 0.9 * np.cos(a) + np.pi) % (2 * np.pi) - np.pi
    y = 0.2 + 0.6 * np.sin(a)
    i = np.arange(1, count + 1, dtype=np.int32)
    one = lambda v: np.array([v], np.int32)
    return dict(xq=x, yq=y, nextq=np.roll(i, -1), indq=one(1), npq=one(count), i1q=one(1),
                i2q=one(count), qjump=1.5)


@pytest.mark.parametrize("n,opts,fp32,nodes", [
    (32, FULL, False, 40), (32, NONE, True, 257), (64, FULL, False, 1000), (128, NONE, False, 333),
    (256, FULL, True, 700), (256, NONE, False, 200_000), (512, FULL, False, 900),
    (512, NONE, False, 0), (1024, FULL, False, 500), (2048, NONE, False, 500),
    # the node update counts crossings 31 nodes a warp, up to 148 * 1024 nodes
    (64, NONE, False, 31), (64, FULL, False, 62), (64, NONE, False, 63),
    (256, NONE, False, 148 * 1024), (256, NONE, False, 148 * 1024 + 1)])
def test_one_advance(oracle_mod, gpu_lib, n, opts, fp32, nodes):
    from hydra_b200.casl import CaslGPU
    kw = dict(ncontq=20, dtmax=0.05, npm=1 << 19, nm=1 << 12, **opts)
    o, g = oracle_mod.Oracle(n, **kw), CaslGPU(n, **kw)
    if fp32:
        g.set_precision(1)
    qs = ptospc_np(random_pv(n, 5.0, 1))
    qd = ptospc_np(random_pv(n, 7.0, 2, rms=0.3))
    for s in (o, g):
        if nodes:
            s.set_contours(ellipse(n, nodes))
        s.set_field("qs", qs)
        s.set_field("qd", qd)
        s.set_scalar("t", 0.0)
        s.set_scalar("twist", 0.0)
        s.advance()
    rel = lambda a, b: np.abs(a - b).max() / np.abs(b).max()
    node_bar, field_bar = (1e-6, 1e-6) if fp32 else (1e-12, 1e-11)
    if nodes:
        co, cg = o.contours(), g.contours()
        for k in ("xq", "yq"):
            assert rel(cg[k], co[k]) < node_bar, k
        assert rel(g.field("qc"), o.field("qc")) < 1e-12
    assert abs(g.scalar("dt") - o.scalar("dt")) <= node_bar * o.scalar("dt")
    for f in ("uu", "vv"):
        assert rel(g.field(f), o.field(f)) < node_bar, f
    for f in ("qs", "qd", "qq", "pp", "emq", "epq"):
        assert rel(g.field(f), o.field(f)) < field_bar, f
    g.close()
    o.close()
