"""casl_con2grid_noalloc leaves its scratch cleared for the next call: calls in
a row on every grid size it serves, before and after a call that reports an
error, against the handle's con2grid.  Both form the same exact integers and
round them the same way, so the fields are equal."""
import ctypes

import numpy as np
import pytest

from hydra_b200.synthetic import random_pv

pytestmark = pytest.mark.gpu


def call(lib, n, c, x, y):
    import torch
    dev = [torch.tensor(a, device="cuda:0") for a in (x, y, np.asarray(c["nextq"], np.int32))]
    qc = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    rc = lib.casl_con2grid_noalloc(n, 2 * np.pi, 2 * np.pi, int(c["nptq"]), float(c["qjump"]),
                                   *[ctypes.c_void_p(a.data_ptr()) for a in dev],
                                   ctypes.c_void_p(qc.data_ptr()), None)
    return rc, qc.cpu().numpy()


@pytest.mark.parametrize("n", [32, 64, 128, 256])
def test_calls_in_a_row(gpu_lib, n):
    from hydra_b200.casl import CaslGPU
    g = CaslGPU(n, ncontq=20)
    g.initialise(random_pv(n, 4.0, n))
    c, ref = g.contours(), g.con2grid()
    x, y = np.array(c["xq"]), np.array(c["yq"])
    for bad in (False, False, True, False, False):
        xb = x.copy()
        if bad:
            xb[len(xb) // 2] = 4.0  # outside the domain: that node is skipped and reported
        rc, q = call(gpu_lib, n, c, xb, y)
        if bad:
            assert rc != 0
        else:
            assert rc == 0 and np.array_equal(q, ref)
    g.close()


@pytest.mark.parametrize("n", [32, 64, 128, 256, 512])
def test_column_widths(oracle_mod, gpu_lib, n):
    """The handle's con2grid with CTAs of 3 (up to 256) and 7 coarse columns
    (512) against the oracle's: the same integers, whose mean the oracle takes
    off in floating point."""
    from hydra_b200.casl import CaslGPU
    o = oracle_mod.Oracle(n, ncontq=20, dtmax=0.05)
    o.initialise(random_pv(n, 4.0, n + 1))
    ref = o.con2grid()
    g = CaslGPU(n, ncontq=20)
    g.set_contours(o.contours())
    q = g.con2grid()
    assert np.abs(q - ref).max() <= 1e-12 * np.abs(ref).max()
    g.close()
    o.close()
