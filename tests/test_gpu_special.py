"""The FP32 tail mass and inverse normal of the mixed-precision step
(csrc/normal32.cuh) against erfc and the normal quantile in float64 on dense
grids of FP32 inputs, and the FP64 step's erf and quantile (normal64.cuh)
against mpmath (needs a B200)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
from scipy.special import erfc, ndtri

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "csrc", "special_unit.cu")
HDRS = [os.path.join(HERE, "..", "dbgenzpaper_b200", "csrc", h) for h in ("normal32.cuh", "normal64.cuh", "normtab.h")]
LIB = os.path.join(HERE, "csrc", "libspecial_unit.so")


def _lib():
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(map(os.path.getmtime, [SRC] + HDRS)):
        subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                        "-Xcompiler", "-fPIC", "-o", LIB, SRC], check=True)
    L = C.CDLL(LIB)
    pf = C.POINTER(C.c_float)
    L.tail_mass_eval.argtypes = [pf, pf, C.c_int]
    L.phi_inv_eval.argtypes = [pf, pf, C.c_int]
    pd = C.POINTER(C.c_double)
    L.f64_eval.argtypes = [pd, pd, C.c_int, C.c_int]
    return L


def test_tail_mass_relative_error():
    L = _lib()
    x = np.linspace(0.0, 9.0, 900001).astype(np.float32)
    out = np.zeros_like(x)
    pf = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))
    assert L.tail_mass_eval(pf(x), pf(out), x.size) == 0
    ref = 0.5 * erfc(x.astype(np.float64))
    rel = np.abs(out.astype(np.float64) / ref - 1.0)
    near = x <= 4.5
    assert rel[near].max() < 3e-6, rel[near].max()
    assert rel.max() < 1.5e-5, rel.max()
    assert out[0] == pytest.approx(0.5, rel=1e-6) and np.all(np.diff(out) <= 0)


def test_phi_inv_lower_relative_error():
    L = _lib()
    p = np.exp(np.linspace(np.log(2.3e-16), np.log(0.5), 2000001)).astype(np.float32)
    p = np.unique(p[(p > 0) & (p <= 0.5)])
    out = np.zeros_like(p)
    pf = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))
    assert L.phi_inv_eval(pf(p), pf(out), p.size) == 0
    ref = ndtri(p.astype(np.float64))
    far = p < 0.45  # away from the zero of Phi^-1 at 1/2
    rel = np.abs(out[far].astype(np.float64) / ref[far] - 1.0)
    assert rel.max() < 5e-7, rel.max()
    assert np.all(np.abs(out[~far] - ref[~far]) < 2e-8 + 5e-7 * np.abs(ref[~far]))
    assert out[-1] == 0.0


def _f64(x, which):
    out = np.zeros_like(x)
    pd = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    assert _lib().f64_eval(pd(x), pd(out), x.size, which) == 0
    return out


def test_erf_f64_absolute_error():
    """erf to 1.2e-16 absolute (half an ulp of 1 from the last rounding, the
    table's rounding and the series): table nodes, midpoints, the end of the
    table, signed zeros and infinities among the points."""
    import mpmath as mp
    a = np.arange(193) / 32.0
    x = np.concatenate([a, a + 1 / 64, np.nextafter(a + 1 / 64, 9), np.random.default_rng(1).uniform(0, 6.2, 4000),
                        [6.0, 6.5, 9.0, 40.0, 1e-300, 5e-17]])
    x = np.concatenate([x, -x, [np.inf, -np.inf]])
    out = _f64(x, 0)
    with mp.workdps(30):
        err = np.array([abs(float(mp.mpf(float(o)) - mp.erf(float(v)))) for o, v in zip(out, x)])
    assert err.max() < 1.5e-16, (err.max(), x[err.argmax()])
    assert np.array_equal(np.abs(out[np.abs(x) >= 6]), np.ones((np.abs(x) >= 6).sum()))


def test_quantile_f64_error():
    """sqrt(2) erfinv(v) to 2 rounding errors (2.2e-16 relative), the table's
    5e-17 absolute in erfc / g and the dropped terms: 4e-16 (|y| + 1/2), over the
    step's range 2^-52 <= 1 - |v|."""
    import mpmath as mp
    rng = np.random.default_rng(2)
    q = np.concatenate([np.exp(rng.uniform(np.log(4.5e-16), 0, 1500)), rng.uniform(0, 1, 1000), 2.0 ** -np.arange(1, 52)])
    v = 1.0 - q
    v = np.concatenate([v, -v, [0.0, 1 - 2.0**-51, -(1 - 2.0**-51), 1e-12, -1e-300]])
    out = _f64(v, 1)
    err = np.zeros(v.size)
    with mp.workdps(30):
        for i, (o, w) in enumerate(zip(out, v)):
            x, w = mp.mpf(float(o)) / mp.sqrt(2), mp.mpf(float(w))
            for _ in range(2):  # from a value right to 1e-15: two Newton steps give 30 digits
                t = mp.erfc(abs(x)) - (1 - abs(w))
                x = mp.sign(w) * (abs(x) + t * mp.sqrt(mp.pi) / 2 * mp.exp(x * x))
            err[i] = abs(float(mp.mpf(float(o)) - mp.sqrt(2) * x)) / (abs(float(o)) + 0.5)
    assert err.max() < 4e-16, (err.max(), v[err.argmax()])
