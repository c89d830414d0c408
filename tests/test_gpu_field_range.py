"""The device's range and l1 norm of initial fields: an ensemble's contour
intervals are exactly (max - min)/ncontq of every member's field, whatever its
sign or size, and a field whose l1 norm lies just below, at or just above the
line under which nothing is contoured takes the oracle's side."""
import numpy as np
import pytest

from hydra_b200.synthetic import random_pv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 64, 256])
def test_member_intervals(gpu_lib, n):
    from hydra_b200.casl import CaslEnsemble
    q = random_pv(n, 4.0, n)
    fields = [q, q + 100.0, q - 100.0, 1e-3 * q, q * 1e3, np.zeros((n, n))]
    levels = [20, 7, 9, 11, 13, 5]
    g = CaslEnsemble(n, len(fields), ncontq=20)
    g.initialise_members(fields, levels)
    for m, (f, k) in enumerate(zip(fields, levels)):
        nq, _, qj = g.member_counts(m)
        assert qj == (f.max() - f.min()) / k
        assert (nq == 0) == (m == 5)
    g.close()


@pytest.mark.parametrize("over", [-1e-6, -1e-12, 0.0, 1e-12, 1e-6, 1.0])
def test_nothing_to_contour(oracle_mod, gpu_lib, over):
    from hydra_b200.casl import CaslGPU
    n = 64
    q = random_pv(n, 4.0, 5)
    q = q * ((1.0 + over) * 1e-12 / ((2 * np.pi / n) ** 2 * np.abs(q).sum()))
    o, g = oracle_mod.Oracle(n, ncontq=20), CaslGPU(n, ncontq=20)
    o.initialise(q)
    g.initialise(q)
    co, cg = o.contours(), g.contours()
    assert (cg["nq"] == 0) == (co["nq"] == 0)
    if abs(over) > 1e-9:
        assert (co["nq"] == 0) == (over < 0)
    o.close()
    g.close()
