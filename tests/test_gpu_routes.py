"""What a call's route through the loops must keep: the working precision of the
conditioning sums, the checkpoint setting of banded gradients, and the
results either side of the loop-choice lines (needs a B200)."""
import ctypes as C

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


def _sparse_problem(D, n, offsets, seed, sobol, m=600, context=None):
    # a factor with entries at the given distances above its diagonal
    rng = np.random.default_rng(seed)
    U = np.eye(n)
    for o in offsets:
        i = np.arange(n - o)
        U[i, i + o] = rng.uniform(-0.6, 0.6, n - o) / np.sqrt(len(offsets))
    S = W.correlation(U.T @ U)
    b = rng.uniform(1.5, 3.5, n)
    pts = _points("Sobol" if sobol else "Richtmyer", n, rng)
    return D.QMCDataSparse(S, np.full(n, -np.inf), b, D.QMC_opts(m=m, n_reps=R, max_pts=m, max_abs_err=0.0),
                           qmc_type="Sobol" if sobol else "Richtmyer", context=context, **pts)


def _state(ctx):
    prof = L.DbgzProfile()
    L.check(L.lib().dbgz_get_profile(ctx.handle, C.byref(prof)), ctx.handle)
    return int(prof.grad_state_bytes), int(prof.grad_chunks)


# set_grad_checkpoints decides the state of any banded gradient, of factors that
# fill their band (the first two) too.  Segments inside, equal to and longer than
# the problem; same bits as the whole state, also with the samples in several
# chunks.
@pytest.mark.parametrize("prec", [L.PREC_FP64, L.PREC_FP32_SIMT])
@pytest.mark.parametrize("n,offsets,seg,sobol", [(150, range(1, 7), 32, False), (300, range(1, 41), 64, True),
                                                 (420, (1, 300), 5, False), (500, (1, 2, 310), 100, True),
                                                 (420, (3, 290), 420, False), (300, (250,), 600, True)])
def test_checkpoint_setting_bounds_the_state(dbgz, prec, n, offsets, seg, sobol):
    D = dbgz
    ctx = D.Context(0)
    try:
        L.lib().dbgz_set_profiling(ctx.handle, 1)
        Q = _sparse_problem(D, n, offsets, n + seg, sobol, context=ctx)
        default = D.qmc_pnorm_grad(Q, precision=prec)
        ctx.set_grad_checkpoints(0)
        full = D.qmc_pnorm_grad(Q, precision=prec)
        state_full, _ = _state(ctx)
        ctx.set_grad_checkpoints(seg)
        ck = D.qmc_pnorm_grad(Q, precision=prec)
        state_ck, chunks = _state(ctx)
        assert chunks == 1
        ctx.set_state_budget(1 << 20)  # several chunks of tiles
        ckc = D.qmc_pnorm_grad(Q, precision=prec)
        assert _state(ctx)[1] > 1
        Q.close()
        if 2 * seg < n and max(offsets) < 64:
            assert state_ck < state_full
        assert state_ck != state_full
        assert ck[0] == full[0] and ck[1] == full[1] and ckc[0] == full[0]
        assert np.array_equal(ck[3], full[3]) and np.array_equal(ck[4], full[4])
        for x, y in zip(ckc[3:5], full[3:5]):
            assert np.linalg.norm(x - y) <= 1e-11 * np.linalg.norm(y)
        # the default may run in another loop: the bars of the other banded tests
        tol = 1e-11 if prec == L.PREC_FP64 else 2e-3
        assert abs(default[0] - full[0]) <= (1e-12 if prec == L.PREC_FP64 else 5e-6 + 2e-5 * full[0])
        for x, y in zip(default[3:5], full[3:5]):
            assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y)
    finally:
        ctx.close()


# either side of the lines between the warp-level and the tcgen05 loop, which
# depend on the pass's tiles of 128 samples per SM (148): up to 2, more than 4 and up
# to 6, and others.  Bars of the split-BF16 mode.
@pytest.mark.parametrize("qmc,n,tiles,grad", [
    ("Richtmyer", 257, 294, False), ("Sobol", 258, 294, False), ("Sobol", 300, 600, False),
    ("Richtmyer", 301, 600, False), ("Richtmyer", 401, 300, False), ("Richtmyer", 170, 6, True),
    ("Richtmyer", 171, 294, True), ("Sobol", 200, 294, True), ("Sobol", 201, 6, True), ("Richtmyer", 301, 600, True),
    ("Sobol", 431, 600, True), ("Sobol", 560, 300, True), ("Sobol", 561, 300, True)])
def test_split_bf16_at_the_lines_by_tiles(dbgz, qmc, n, tiles, grad):
    D = dbgz
    rng = np.random.default_rng(n)
    S = W.correlation(W.rand_spd(n, 1.0, rng))
    a, b = W.bounds_quarter(S)
    pts = _points(qmc, n, rng)
    m = 128 * tiles // R - 5
    out = {}
    for prec in (L.PREC_FP64, L.PREC_FP32_SPLIT_BF16):
        Q = D.QMCData(S, a, b, D.QMC_opts(m=m, n_reps=R, max_pts=m, max_abs_err=0.0), qmc_type=qmc, **pts)
        out[prec] = D.qmc_pnorm_grad(Q, precision=prec) if grad else D.qmc_pnorm(Q, precision=prec)
        Q.close()
    r64, r = out[L.PREC_FP64], out[L.PREC_FP32_SPLIT_BF16]
    assert abs(r[0] - r64[0]) <= 5e-6 + 2e-5 * abs(r64[0])
    for x, y in zip(r[3:6], r64[3:6]) if grad else ():
        assert np.linalg.norm(x - y) <= 2e-3 * np.linalg.norm(y)


# the line looks at the whole pass: sample chunks small enough for another one
# give the same estimate to the last bit
def test_sample_chunks_take_the_pass_s_loop(dbgz):
    D = dbgz
    n, m = 350, 12800  # 300 tiles
    rng = np.random.default_rng(n)
    S = W.correlation(W.rand_spd(n, 1.0, rng))
    a, b = W.bounds_quarter(S)
    ctx = D.Context(0)
    try:
        Q = D.QMCData(S, a, b, D.QMC_opts(m=m, n_reps=R, max_pts=m, max_abs_err=0.0), context=ctx,
                      **_points("Richtmyer", n, rng))
        one = D.qmc_pnorm_grad(Q, precision=L.PREC_FP32_SPLIT_BF16)
        ctx.set_state_budget(100 << 20)
        two = D.qmc_pnorm_grad(Q, precision=L.PREC_FP32_SPLIT_BF16)
        chunks = _state(ctx)[1]
        Q.close()
        assert chunks > 1 and one[0] == two[0] and one[1] == two[1]
        for x, y in zip(two[3:6], one[3:6]):
            assert np.linalg.norm(x - y) <= 1e-6 * np.linalg.norm(y)
    finally:
        ctx.close()
