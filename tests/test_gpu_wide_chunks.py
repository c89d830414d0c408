"""Contours so many and so close that 16 neighbouring fine-grid edges meet more
than 65535 of them, the most that 16-bit places inside such a chunk number:
recontouring them against the oracle (topology identical; nodes 1e-8, the bar of
a recontouring from contours)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def strips(n, levels, per_cell, cols, axis):
    """`levels` contours around each of `per_cell` strips one fine cell wide: the
    level goes up and down at every fine line across them."""
    fine = 2 * np.pi / (16 * n)
    # half a fine cell off the grid lines across, a quarter off them along
    along = -np.pi + fine * (np.linspace(64, 64 + cols, 6) + 0.25)
    xs, ys = [], []
    for s in range(per_cell):
        c = -np.pi + fine * (16 * 5 + 2 * s + 1)
        u = np.concatenate([along, along[::-1]])
        v = np.concatenate([np.full(6, c - 0.5 * fine), np.full(6, c + 0.5 * fine)])
        x, y = (u, v) if axis == "x" else (v[::-1], u[::-1])
        xs.append(x), ys.append(y)
    x, y = np.tile(np.concatenate(xs), levels), np.tile(np.concatenate(ys), levels)
    m = per_cell * levels
    i1q = (1 + 12 * np.arange(m)).astype(np.int32)
    nextq = np.arange(2, 12 * m + 2, dtype=np.int32)
    nextq[11::12] = i1q
    return dict(xq=x, yq=y, nextq=nextq, indq=np.repeat(np.arange(1, levels + 1), per_cell).astype(np.int32),
                npq=np.full(m, 12, np.int32), i1q=i1q, i2q=(i1q + 11).astype(np.int32), qjump=0.01)


@pytest.mark.parametrize("axis,levels", [("x", 4200), ("y", 4200), ("x", 4095)])
def test_recontour(oracle_mod, gpu_lib, axis, levels):
    from hydra_b200.casl import CaslGPU
    n = 32
    c = strips(n, levels, 8, 32, axis)
    kw = dict(ncontq=100, nlevm=20000, npm=1 << 22, nm=1 << 17)
    o, g = oracle_mod.Oracle(n, **kw), CaslGPU(n, **kw)
    for s in (o, g):
        s.set_contours(c)
        s.recontour(np.zeros((n, n)))
    co, cg = o.contours(), g.contours()
    assert (cg["nq"], cg["nptq"]) == (co["nq"], co["nptq"])
    assert co["nq"] >= 8 * levels - 16
    for k in ("npq", "i1q", "i2q", "indq", "nextq"):
        assert np.array_equal(cg[k], co[k]), k
    for k in ("xq", "yq"):
        assert np.abs(cg[k] - co[k]).max() < 1e-8, k
    g.close()
    o.close()
