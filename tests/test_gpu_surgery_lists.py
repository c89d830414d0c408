"""Surgery's box lists where segments and boxes are unlike a smooth flow's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASL_ECAPACITY, CASL_EDOMAIN = 2, 5


def one_level(parts):
    """Closed contours of one level, from their nodes' (x, y)."""
    npq = np.array([len(x) for x, _ in parts], np.int32)
    i2q = np.cumsum(npq).astype(np.int32)
    i1q = i2q - npq + 1
    nextq = np.arange(2, i2q[-1] + 2, dtype=np.int32)
    nextq[i2q - 1] = i1q
    x, y = (np.concatenate([p[k] for p in parts]) for k in (0, 1))
    return dict(xq=x, yq=y, nextq=nextq, indq=np.ones(len(parts), np.int32), npq=npq, i1q=i1q,
                i2q=i2q, qjump=1.0)


def test_more_entries_than_an_int_counts(gpu_lib):
    """A contour back and forth over half the domain: its segments lie in more
    than 2^31 boxes together, which must end in the capacity error and not in
    a count that has wrapped around."""
    from hydra_b200.casl import CaslError, CaslGPU
    n, count = 2048, 90_000
    rng = np.random.default_rng(1)
    side = np.where(np.arange(count) % 2 == 0, -1.5, 1.5)
    x, y = side + rng.uniform(-0.05, 0.05, count), side + rng.uniform(-0.05, 0.05, count)
    # the boxes its segments span (1.2 sqrt(nodes) a side), less four each
    nb = round(1.2 * count ** 0.5)
    bx, by = (np.floor(nb + nb / (2 * np.pi) * (v + np.pi)).astype(np.int64) for v in (x, y))
    span = lambda b: np.abs(np.diff(np.append(b, b[0]))) + 1
    assert (span(bx) * span(by) - 4).sum() > 1.1 * 2**31
    g = CaslGPU(n, ncontq=20, npm=1 << 18, nm=1 << 12)
    c = one_level([(x, y)])
    g.set_contours(c)
    with pytest.raises(CaslError) as e:
        g.surgery()
    assert e.value.code == CASL_ECAPACITY
    # nothing outside the lists was written: a small state's surgery is right
    a = 2 * np.pi * np.arange(300) / 300
    g.set_contours(one_level([(np.cos(a), np.sin(a))]))
    g.surgery()
    assert g.counts()[0] == 1
    g.close()


def test_nodes_that_are_not_finite(gpu_lib):
    """Surgery called on what a failed step left (nodes that are NaN have no
    box) ends in the domain error and writes nowhere it should not: the next
    state's surgery is that of a fresh handle."""
    from hydra_b200.casl import CaslError, CaslGPU
    from hydra_b200.synthetic import random_pv
    kw = dict(ncontq=20, dtmax=0.05, npm=1 << 18, nm=1 << 14)
    g, f = CaslGPU(64, **kw), CaslGPU(64, **kw)
    for s in (g, f):
        s.initialise(random_pv(64, 5.0, 3))
    good = f.contours()
    qs = g.field("qs")
    qs[2, 3] = np.nan
    g.set_field("qs", qs)
    for call in (g.step, g.surgery):
        with pytest.raises(CaslError) as e:
            call()
        assert e.value.code == CASL_EDOMAIN
    for s in (g, f):
        s.set_contours(good)
        s.surgery()
    cg, cf = g.contours(), f.contours()
    for k in ("nq", "nptq", "xq", "yq", "nextq"):
        assert np.array_equal(cg[k], cf[k]), k
    g.close()
    f.close()
