"""Renode's one-pass density sums and counts (k_rn_nodes, k_rn_contours) and its
placement (k_rn_place) at the edges of their tiles (1792 nodes and others, 256
contours), against the oracle: contours one node below, at and above a tile, a
contour over many tiles at each of the tile sizes, one with a corner at every
other node (pieces across tiles), and a state of many small contours through a
surgery.

Bars: node counts identical, positions 1e-12 (the bars of the renode and
surgery tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TILE = 1792


def ring(m, r, wob, k):
    a = 2 * np.pi * np.arange(m) / m
    rr = r * (1 + wob * np.cos(k * a))
    return rr * np.cos(a) + 0.1, rr * np.sin(a) - 0.2


@pytest.mark.parametrize("m,zigzag", [(4, 0), (27, 0), (29, 0), (TILE - 1, 0), (TILE, 0), (TILE + 1, 0),
                                      (9 * TILE + 5, 0), (60_000, 0), (TILE, 1), (3 * TILE + 2, 1),
                                      (2 * TILE, 200), (400_001, 50), (1_100_003, 0), (1_100_003, 300)])
def test_one_contour(oracle_mod, gpu_lib, m, zigzag):
    from hydra_b200.casl import CaslGPU
    o, g = oracle_mod.Oracle(64, ncontq=20), CaslGPU(64, ncontq=20)
    x, y = ring(m, 1.1, 0.3, 7)
    if zigzag:  # teeth: two corners every 2*zigzag nodes
        f = 1 + 0.2 * ((np.arange(m) // zigzag) % 2)
        x, y = x * f, y * f
    xo, yo = o.renode(x, y)
    xg, yg = g.renode(x, y)
    assert len(xg) == len(xo)
    # the oracle adds m densities one after the other, so a node may move by
    # m * 2**-53 of the contour's length, which passes the bar for the longest
    length = np.hypot(np.diff(x, append=x[0]), np.diff(y, append=y[0])).sum()
    bar = 1e-12 * np.pi if m <= 60_000 else m * 2.0**-53 * length
    assert np.abs(xg - xo).max() <= bar and np.abs(yg - yo).max() <= bar
    g.close()
    o.close()


@pytest.mark.parametrize("count", [1, 255, 256, 257, 900, 1023, 1024, 1025, 2500])
def test_many_contours(oracle_mod, gpu_lib, count):
    from hydra_b200.casl import CaslGPU
    rng = np.random.default_rng(count)
    xs, ys, npq = [], [], []
    side = int(np.ceil(np.sqrt(count)))
    for j in range(count):
        m = int(rng.integers(5, 60))
        x, y = ring(m, 2.2 / side, 0.2, 3)
        xs.append(x - 0.1 - 3.0 + 6.0 * (j % side + 0.5) / side)
        ys.append(y + 0.2 - 3.0 + 6.0 * (j // side + 0.5) / side)
        npq.append(m)
    npq = np.array(npq, np.int32)
    i1 = np.concatenate([[1], 1 + np.cumsum(npq)[:-1]]).astype(np.int32)
    i2 = (i1 + npq - 1).astype(np.int32)
    nxt = np.arange(2, npq.sum() + 2, dtype=np.int32)
    nxt[i2 - 1] = i1
    c = dict(xq=np.concatenate(xs), yq=np.concatenate(ys), nextq=nxt, npq=npq, i1q=i1, i2q=i2,
             indq=np.sort(rng.integers(-3, 4, count)).astype(np.int32), qjump=0.7)
    o, g = oracle_mod.Oracle(64, ncontq=20), CaslGPU(64, ncontq=20)
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


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_box_lists(oracle_mod, gpu_lib, seed):
    """Surgery's box lists: one level of 200 small rings close enough to be
    joined, hundreds of segments in a box, and a coarse ring through them whose
    segments each cross a hundred boxes.  Some ring nodes lie just below the
    edge of a box: there the box they are tested in is not among their
    segment's (see the last assertion on the inputs)."""
    from hydra_b200.casl import CaslGPU
    rng = np.random.default_rng(seed)
    dm = 0.04 * 6.25 * (2 * np.pi / 64) / 4
    xs, ys, npq = [], [], []
    for j in range(200):
        x, y = ring(100, 0.02, 0.1, 3)
        xs.append(x - 0.1 + 2.0 * np.cos(j // 2) + (j % 2) * (0.04 + 0.3 * dm))
        ys.append(y + 0.2 + 2.0 * np.sin(j // 2) + rng.uniform(-0.2, 0.2) * dm)
        npq.append(100)
    x, y = ring(24, 2.0, 0.02, 5)
    xs.append(x - 0.1), ys.append(y + 0.2), npq.append(24)
    npq = np.array(npq, np.int32)
    x, y = np.concatenate(xs), np.concatenate(ys)
    nbx = float(int(1.2 * np.sqrt(float(npq.sum())) + 0.5))
    b = nbx / (2 * np.pi)
    edge = 0
    for i in range(0, 20_000, 7):
        xe = -np.pi + (np.floor(b * (x[i] + np.pi)) + 1) / b
        for _ in range(8):
            if np.floor(b * (xe + np.pi)) + nbx < np.floor(nbx + b * (xe + np.pi)):
                break
            xe = np.nextafter(xe, -4)
        else:
            continue
        if abs(xe - x[i]) < 2e-3:
            x[i], edge = xe, edge + 1
    i1 = np.concatenate([[1], 1 + np.cumsum(npq)[:-1]]).astype(np.int32)
    i2 = (i1 + npq - 1).astype(np.int32)
    nxt = np.arange(2, npq.sum() + 2, dtype=np.int32)
    nxt[i2 - 1] = i1
    c = dict(xq=x, yq=y, nextq=nxt, npq=npq, i1q=i1, i2q=i2, indq=np.ones(201, np.int32), qjump=0.7)
    assert edge > 0
    o, g = oracle_mod.Oracle(64, ncontq=20), CaslGPU(64, ncontq=20)
    for s in (o, g):
        s.set_contours(c)
        s.surgery()
    co, cg = o.contours(), g.contours()
    assert co["nq"] != 201 and (cg["nq"], cg["nptq"]) == (co["nq"], co["nptq"])
    for k in ("npq", "i1q", "i2q", "indq", "nextq"):
        assert np.array_equal(cg[k], co[k]), k
    for k in ("xq", "yq"):
        assert np.abs(cg[k] - co[k]).max() <= 1e-12 * np.pi, k
    g.close()
    o.close()
