"""The sample loops, their dispatch rules and the pivoted factorisation at the
sizes where tiles, groups, chunks and rings end (needs a B200).

Bars, as elsewhere: FP64 replicate means within 1e-12 relative of the oracle;
FP32 probabilities within 5e-6 + 2e-5 P of FP64 on the same points; FP32
gradients within 2e-3 of FP64 in norm; FP64 gradients against a central
difference of step 1e-6 along all upper bounds (rounding 1e-16 / 1e-6,
truncation 1e-12: within 2e-6 of the larger of the derivative and P);
factors bit for bit."""
import numpy as np
import pytest

from dbgenzpaper_b200 import _lib as L
from dbgenzpaper_b200 import workloads as W

pytestmark = pytest.mark.gpu
R = 3
NAMES = ["Richtmyer", "Sobol"]


@pytest.fixture(scope="module")
def D(dbgz):
    dbgz.get_context(0)
    return dbgz


def _points(qmc, n, rng):
    if qmc == "Richtmyer":
        return {"shifts": rng.random((n - 1, R))}
    return {"ushifts": rng.integers(0, 2**64, size=(n - 1, R), dtype=np.uint64)}


def _oracle(D, oracle, Q, qmc, pts, m, sparse):
    kw = dict(m=m, n_reps=R, max_pts=m, max_abs_err=0.0, sparse=sparse)
    if qmc == "Richtmyer":
        kw["shifts"] = pts["shifts"]
    else:
        kw.update(qmc_type=oracle.SOBOL, V=D.sobol_dirnums(Q.C.U.shape[0] - 1), ushifts=pts["ushifts"],
                  sobol_first=Q.sobol_first)
    F = Q.C
    return oracle.qmc_pnorm(F.U, F.a, F.b, **kw)


def _opts(D, m):
    return D.QMC_opts(m=m, n_reps=R, max_pts=m, max_abs_err=0.0)


def _bounds(n, rng, upper):
    a = np.full(n, -np.inf) if upper else rng.uniform(-2.5, -0.2, n)
    return a, rng.uniform(0.2, 2.5, n)


# m = 200: a full tile of 128 samples and one of 72
@pytest.mark.parametrize("qmc", NAMES)
@pytest.mark.parametrize("n", [2, 3, 9, 10, 31, 32, 33, 34, 41, 64, 65, 66, 97])
def test_dense_loops_at_group_edges(D, oracle, n, qmc):
    rng = np.random.default_rng(n)
    S = W.correlation(W.rand_spd(n, 1.0, rng))
    a, b = _bounds(n, rng, n % 2 == 0)
    pts = _points(qmc, n, rng)
    Q = D.QMCData(S, a, b, _opts(D, 200), qmc_type=qmc, **pts)
    r64 = D.qmc_pnorm(Q, precision=L.PREC_FP64, return_reps=True)
    rc = _oracle(D, oracle, Q, qmc, pts, 200, False)
    np.testing.assert_allclose(r64[3], rc[3], rtol=1e-12)
    for prec in (L.PREC_FP32_SPLIT_BF16, L.PREC_FP32_SIMT):
        Q.close()
        Q = D.QMCData(S, a, b, _opts(D, 200), qmc_type=qmc, **pts)
        P = D.qmc_pnorm(Q, precision=prec)[0]
        assert abs(P - rc[0]) <= 5e-6 + 2e-5 * abs(rc[0])
    Q.close()


# fewer bits than the staged words hold: their entries are cut to n_bits
@pytest.mark.parametrize("n_bits", [1, 12, 31])
def test_staged_integers_cut_to_n_bits(D, oracle, n_bits):
    n, m = 70, 200
    rng = np.random.default_rng(n_bits)
    S = W.correlation(W.rand_spd(n, 1.0, rng))
    a, b = _bounds(n, rng, False)
    us = rng.integers(0, 2**n_bits, size=(n - 1, R), dtype=np.uint64)
    opts = D.QMC_opts(m=m, n_reps=R, max_pts=m, max_abs_err=0.0, n_bits=n_bits)
    Q = D.QMCData(S, a, b, opts, qmc_type="Sobol", ushifts=us)
    reps = D.qmc_pnorm(Q, precision=L.PREC_FP64, return_reps=True)[3]
    F = Q.C
    rc = oracle.qmc_pnorm(F.U, F.a, F.b, m=m, n_reps=R, max_pts=m, max_abs_err=0.0, qmc_type=oracle.SOBOL,
                          V=D.sobol_dirnums(n - 1), ushifts=us, sobol_first=Q.sobol_first, n_bits=n_bits)
    np.testing.assert_allclose(reps, rc[3], rtol=1e-12)
    Q.close()


# either side of the lines between the warp-level and the tcgen05 loop
@pytest.mark.parametrize("qmc,n,grad", [("Richtmyer", 400, False), ("Sobol", 401, False), ("Richtmyer", 430, True),
                                        ("Richtmyer", 431, True), ("Sobol", 600, True), ("Sobol", 601, True)])
def test_split_bf16_at_the_loops_line(D, qmc, n, grad):
    rng = np.random.default_rng(n)
    S = W.correlation(W.rand_spd(n, 1.0, rng))
    a, b = W.bounds_quarter(S)
    pts = _points(qmc, n, rng)
    out = {}
    for prec in (L.PREC_FP64, L.PREC_FP32_SPLIT_BF16):
        Q = D.QMCData(S, a, b, _opts(D, 200), qmc_type=qmc, **pts)
        out[prec] = D.qmc_pnorm_grad(Q, precision=prec) if grad else D.qmc_pnorm(Q, precision=prec)
        Q.close()
    r64, r = out[L.PREC_FP64], out[L.PREC_FP32_SPLIT_BF16]
    assert abs(r[0] - r64[0]) <= 5e-6 + 2e-5 * abs(r64[0])
    for x, y in zip(r[3:6], r64[3:6]) if grad else ():
        assert np.linalg.norm(x - y) <= 2e-3 * np.linalg.norm(y)


def _band_data(D, n, band, qmc, pts, a, b, m=200):
    i = np.arange(n)
    S = 0.85 ** np.abs(i[:, None] - i[None, :]) * (1 + 0.1 * np.cos(i[:, None]) * np.cos(i[None, :]))
    S = W.correlation(S + 0.05 * np.eye(n))
    Q = D.QMCDataSparse(S, a, b, _opts(D, m), qmc_type=qmc, **pts)
    Q.truncate_band(band)
    return Q


# bands inside one group, at its multiples, longer than the ring's slack, and
# as wide as the problem
@pytest.mark.parametrize("qmc", NAMES)
@pytest.mark.parametrize("n,band", [(2, 1), (33, 1), (34, 33), (65, 31), (97, 32), (98, 33), (300, 7), (200, 64),
                                    (180, 100)])
def test_band_loops_at_group_and_ring_edges(D, oracle, n, band, qmc):
    rng = np.random.default_rng(1000 * n + band)
    a, b = _bounds(n, rng, band % 2 == 0)
    b += 0.5
    pts = _points(qmc, n, rng)
    Q = _band_data(D, n, band, qmc, pts, a, b)
    P, _, _, reps = D.qmc_pnorm(Q, precision=L.PREC_FP64, return_reps=True)
    rc = _oracle(D, oracle, Q, qmc, pts, 200, True)
    np.testing.assert_allclose(reps, rc[3], rtol=1e-12, atol=1e-300)
    Q.close()
    Q = _band_data(D, n, band, qmc, pts, a, b)
    assert abs(D.qmc_pnorm(Q, precision=L.PREC_FP32_SIMT)[0] - P) <= 5e-6 + 2e-5 * abs(P)
    g64 = D.qmc_pnorm_grad(Q, precision=L.PREC_FP64)
    g32 = D.qmc_pnorm_grad(Q, precision=L.PREC_FP32_SIMT)
    Q.close()
    for x, y in zip(g32[3:5], g64[3:5]):
        assert np.linalg.norm(x - y) <= 2e-3 * np.linalg.norm(y)
    h, Ph = 1e-6, []
    for s in (h, -h):
        Q = _band_data(D, n, band, qmc, pts, a, b + s)
        Ph.append(D.qmc_pnorm(Q, precision=L.PREC_FP64)[0])
        Q.close()
    fd = (Ph[0] - Ph[1]) / (2 * h)
    assert abs(g64[4].sum() - fd) <= 2e-6 * max(abs(fd), abs(P)) + 1e-12


# pairs far apart: few entries for the bandwidth, which the CSC loop takes;
# (256, 240) has one checkpoint segment, (600, 400) several
@pytest.mark.parametrize("qmc", NAMES)
@pytest.mark.parametrize("n,dist", [(256, 240), (600, 400)])
def test_few_entries_in_a_wide_band(D, oracle, n, dist, qmc):
    rng = np.random.default_rng(n)
    S = np.eye(n)
    for i in range(0, n - dist, 2):
        S[i, i + dist] = S[i + dist, i] = 0.5
    a, b = np.full(n, -np.inf), rng.uniform(2.0, 4.0, n)
    pts = _points(qmc, n, rng)

    def data(b):
        Q = D.QMCDataSparse(S, a, b, _opts(D, 200), qmc_type=qmc, **pts)
        Q.truncate_band(dist)
        return Q

    Q = data(b)
    P, _, _, reps = D.qmc_pnorm(Q, precision=L.PREC_FP64, return_reps=True)
    rc = _oracle(D, oracle, Q, qmc, pts, 200, True)
    np.testing.assert_allclose(reps, rc[3], rtol=1e-12, atol=1e-300)
    Q.close()
    Q = data(b)
    assert abs(D.qmc_pnorm(Q, precision=L.PREC_FP32_SIMT)[0] - P) <= 5e-6 + 2e-5 * abs(P)
    g64 = D.qmc_pnorm_grad(Q, precision=L.PREC_FP64)
    g32 = D.qmc_pnorm_grad(Q, precision=L.PREC_FP32_SIMT)
    Q.close()
    assert np.linalg.norm(g32[4] - g64[4]) <= 2e-3 * np.linalg.norm(g64[4])
    h, Ph = 1e-6, []
    for s in (h, -h):
        Q = data(b + s)
        Ph.append(D.qmc_pnorm(Q, precision=L.PREC_FP64)[0])
        Q.close()
    fd = (Ph[0] - Ph[1]) / (2 * h)
    assert abs(g64[4].sum() - fd) <= 2e-6 * max(abs(fd), abs(P)) + 1e-12


# the state's tiles, the factor-gradient product's tiles and k ranges
@pytest.mark.parametrize("qmc", NAMES)
@pytest.mark.parametrize("n", [2, 33, 34, 65, 97, 130])
def test_fp64_gradient_at_tile_edges(D, n, qmc):
    rng = np.random.default_rng(n + 7)
    S = W.correlation(W.rand_spd(n, 1.0, rng))
    a, b = _bounds(n, rng, n % 2 == 1)
    pts = _points(qmc, n, rng)

    def data(b):
        return D.QMCData(S, a, b, _opts(D, 200), qmc_type=qmc, **pts)

    Q = data(b)
    P, _, _, da, db, dU = D.qmc_pnorm_grad(Q, precision=L.PREC_FP64)
    g32 = D.qmc_pnorm_grad(Q, precision=L.PREC_FP32_SIMT)
    Q.close()
    for x, y in zip(g32[3:6], (da, db, dU)):
        assert np.linalg.norm(x - y) <= 2e-3 * np.linalg.norm(y)
    h, Ph = 1e-6, []
    for s in (h, -h):
        Q = data(b + s)
        Ph.append(D.qmc_pnorm(Q, precision=L.PREC_FP64)[0])
        Q.close()
    fd = (Ph[0] - Ph[1]) / (2 * h)
    assert abs(db.sum() - fd) <= 2e-6 * max(abs(fd), abs(P)) + 1e-12


# panels of 1 to 512 rows and columns, blocks that end inside a warp
@pytest.mark.parametrize("n,bs1,bs2", [(2, 64, 512), (3, 1, 2), (63, 64, 512), (65, 64, 512), (129, 64, 128),
                                       (200, 64, 64), (257, 33, 256), (512, 64, 512), (513, 64, 512), (520, 128, 512)])
def test_pivoted_factor_at_panel_edges(D, oracle, n, bs1, bs2):
    rng = np.random.default_rng(n + bs1)
    S = W.rand_spd(n, 1.0, rng)
    a, b = _bounds(n, rng, False)
    a[::7] = -np.inf
    G = D.cholesky_genz(S, a, b, bs1, bs2)
    F = oracle.cholesky_genz(S, a, b, bs1, bs2)
    assert G.rank == F["rank"]
    assert np.array_equal(G.perm, F["perm"]) and np.array_equal(G.U, F["U"])
    assert np.array_equal(G.a, F["a"]) and np.array_equal(G.b, F["b"])
