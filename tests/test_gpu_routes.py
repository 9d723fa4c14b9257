"""What a call's route through the loops must keep (needs a B200)."""
import numpy as np
import pytest

from dbgenzpaper_b200 import _lib as L
from dbgenzpaper_b200 import workloads as W

pytestmark = pytest.mark.gpu
R = 3


def _points(qmc, n, rng):
    if qmc == "Richtmyer":
        return {"shifts": rng.random((n - 1, R))}
    return {"ushifts": rng.integers(0, 2**64, size=(n - 1, R), dtype=np.uint64)}


# The split-BF16 mode's products within a group of 32 variables are FP32.  One
# variable drives the others (its bounds are the tightest, so that it comes
# first): every conditioning sum has one term, s = u y with |s| <= 1.33, which an
# FP32 loop rounds once (2^-24 |s|).  log dc moves by at most phi(0.54) / Phi(0.54)
# / 0.31 = 1.6 times that, over 31 variables: 31 * 1.6 * 1.33 * 2^-24 = 3.9e-6
# between two FP32 loops.  Two BF16 parts (2^-18 of each operand and of their
# product) would move it by up to 6e-4.
@pytest.mark.parametrize("qmc", ["Richtmyer", "Sobol"])
@pytest.mark.parametrize("n", [18, 33])
def test_products_within_a_group_are_fp32(dbgz, n, qmc):
    D = dbgz
    rng = np.random.default_rng(n)
    u = rng.uniform(0.9, 0.95, n)
    u[0] = 1.0
    S = np.outer(u, u)
    np.fill_diagonal(S, 1.0)
    a, b = np.full(n, -1.5), np.full(n, 1.5)
    a[0], b[0] = -1.4, 1.4
    pts = _points(qmc, n, rng)
    lw = {}
    for prec in (L.PREC_FP32_SIMT, L.PREC_FP32_SPLIT_BF16):
        Q = D.QMCData(S, a, b, D.QMC_opts(m=500, n_reps=R, max_pts=500, max_abs_err=0.0), qmc_type=qmc, **pts)
        lw[prec] = D.qmc_pnorm_logw(Q, precision=prec)[0]
        Q.close()
    assert np.abs(lw[L.PREC_FP32_SPLIT_BF16] - lw[L.PREC_FP32_SIMT]).max() <= 4e-6
