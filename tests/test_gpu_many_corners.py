"""Renode of contours with many corners (k_rn_contours): up to 64 pieces a thread
takes a contour, from 65 on the block does, 256 pieces at a time.  Against the
oracle: node counts identical, positions 1e-12 of the domain's half side, or,
where that is more, the rounding of the oracle's running sum of m densities
(m 2^-53 of the contour's length)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def teeth(m, r=1.0, x0=0.0, y0=0.0, depth=0.3):
    """A ring of m teeth: a corner at each of its 2 m nodes."""
    a = np.pi * np.arange(2 * m) / m
    rr = r * (1 + depth * (np.arange(2 * m) % 2))
    return x0 + rr * np.cos(a), y0 + rr * np.sin(a)


def state(parts, levels):
    npq = np.array([len(x) for x, _ in parts], np.int32)
    i2q = np.cumsum(npq).astype(np.int32)
    i1q = i2q - npq + 1
    nextq = np.arange(2, i2q[-1] + 2, dtype=np.int32)
    nextq[i2q - 1] = i1q
    x, y = (np.concatenate([p[k] for p in parts]) for k in (0, 1))
    return dict(xq=x, yq=y, nextq=nextq, indq=np.asarray(levels, np.int32), npq=npq, i1q=i1q, i2q=i2q,
                qjump=1.0)


@pytest.mark.parametrize("m", [31, 32, 33, 127, 128, 129, 500, 20_000])
def test_one_contour(oracle_mod, gpu_lib, m):
    from hydra_b200.casl import CaslGPU
    o, g = oracle_mod.Oracle(64, ncontq=20), CaslGPU(64, ncontq=20)
    x, y = teeth(m)
    xo, yo = o.renode(x, y)
    xg, yg = g.renode(x, y)
    assert len(xg) == len(xo)
    length = np.hypot(np.diff(x, append=x[0]), np.diff(y, append=y[0])).sum()
    bar = max(1e-12 * np.pi, 2 * m * 2.0**-53 * length)
    assert np.abs(xg - xo).max() <= bar and np.abs(yg - yo).max() <= bar
    g.close()
    o.close()


def test_contours_of_a_tile(oracle_mod, gpu_lib):
    """Long and short ones among the 256 of a tile and across two."""
    from hydra_b200.casl import CaslGPU
    rng = np.random.default_rng(2)
    parts = []
    for j in range(300):
        m = int(rng.choice([4, 5, 31, 32, 33, 40])) if j % 3 else 6
        parts.append(teeth(m, 0.12, -2.8 + 0.3 * (j % 19), -2.6 + 0.3 * (j // 19)))
    c = state(parts, np.arange(1, 301))
    o, g = oracle_mod.Oracle(1024, ncontq=20), CaslGPU(1024, ncontq=20, npm=1 << 18, nm=1 << 12)
    for s in (o, g):
        s.set_contours(c)
        s.surgery()
    co, cg = o.contours(), g.contours()
    assert (cg["nq"], cg["nptq"]) == (co["nq"], co["nptq"])
    for k in ("npq", "i1q", "i2q", "indq", "nextq"):
        assert np.array_equal(cg[k], co[k]), k
    for k in ("xq", "yq"):
        assert np.abs(cg[k] - co[k]).max() <= 1e-12 * np.pi, k
    g.close()
    o.close()


def test_two_million_corners(gpu_lib):
    """A contour of 2.2 million corners before 300 others: the tiles of contours
    behind it wait for its count, and that wait has a limit of a second."""
    from hydra_b200.casl import CaslGPU
    per, rows = 12_000, 184
    x1 = -3.0 + 5e-4 * np.arange(per)
    xs = [x1 if r % 2 == 0 else x1[::-1] for r in range(rows)]
    ys = [-1.0 + 5e-3 * r + 1.5e-3 * (np.arange(per) % 2) for r in range(rows)]
    parts = [(np.concatenate(xs), np.concatenate(ys))]
    a = 2 * np.pi * np.arange(40) / 40
    parts += [(-2.8 + 0.2 * (j % 25) + 0.05 * np.cos(a), 0.5 + 0.2 * (j // 25) + 0.05 * np.sin(a))
              for j in range(300)]
    g = CaslGPU(2048, ncontq=20, npm=1 << 23, nm=1 << 12)
    c, best = state(parts, [1] + [2] * 300), 1e9
    for _ in range(3):  # (the first one allocates its scratch)
        g.set_contours(c)
        t = time.perf_counter()
        g.surgery()
        best = min(best, time.perf_counter() - t)
        assert g.counts()[0] == 301 and g.counts()[1] > 2_200_000
    assert best < 0.2, best  # (a second and more with a thread a contour)
    g.close()
