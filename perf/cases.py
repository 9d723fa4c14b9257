"""The work a user has this library do, as cases that can be timed and checked.

Kinds of case (the public calls of ``dbgenzpaper_b200``):

* ``call``    a probability from its inputs: QMCData (upload, pivoted factorisation) and qmc_pnorm;
* ``pass``    qmc_pnorm on a problem that is already factorised;
* ``grad``    P, dP/da, dP/db and dP/dSigma (qmc_pnorm_grad_sigma);
* ``batch``   many small problems of uneven dimension through one BatchPlan;
* ``banded``  qmc_pnorm on a QMCDataSparse whose factor is cut to a band;
* ``banded_grad``  its P, dP/da and dP/db (qmc_pnorm_grad).

``dtype`` is the working type T of QMC_opts: float64 is the default, float32
the mixed-precision path.  A call's numbers are handed on in T, as the
Julia package's qmc_pnorm! returns them in the type of its options.  The
estimate and its error bar are one array, [P, 3 SEM].
"""
import math

import numpy as np
import torch

import dbgenzpaper_b200 as D

SQRT2 = math.sqrt(2.0)


def listed():
    return [
        # the smallest calls: d = 10, where latency and launches count (10^4 lattice points x 10 shifts)
        dict(name="call_f64_d10", kind="call", dtype="float64", d=10, m=10_000, reps=10, qmc="Richtmyer",
             bounds="upper", cov="random"),
        # an ordinary call with every option at its default (Float64, 10^4 points x 12 shifts), two-sided bounds
        dict(name="call_f64_d100", kind="call", dtype="float64", d=100, m=10_000, reps=12, qmc="Richtmyer",
             bounds="finite", cov="random"),
        # a Float64 pass at the dimension of the d = 500 benchmark, Sobol points
        dict(name="pass_f64_d500_sobol", kind="pass", dtype="float64", d=500, m=2**14, reps=12, qmc="Sobol",
             bounds="finite", cov="random"),
        # a whole Float32 call at d = 1000 with the default point count: the factorisation counts
        dict(name="call_f32_d1000", kind="call", dtype="float32", d=1000, m=10_000, reps=12, qmc="Richtmyer",
             bounds="finite", cov="factor"),
        # the largest pass: the d = 1000 factor-model benchmark's size, one-sided bounds
        dict(name="pass_f32_d1000", kind="pass", dtype="float32", d=1000, m=2**17, reps=16, qmc="Richtmyer",
             bounds="upper", cov="factor"),
        # the d = 500 benchmark's size: Sobol points, two-sided bounds
        dict(name="pass_f32_d500_sobol", kind="pass", dtype="float32", d=500, m=2**16, reps=12, qmc="Sobol",
             bounds="finite", cov="random"),
        # sensitivities of a large model (forward, adjoint, factor gradient, Cholesky adjoint)
        dict(name="grad_f32_d1000", kind="grad", dtype="float32", d=1000, m=2**15, reps=16, qmc="Richtmyer",
             bounds="upper", cov="factor"),
        # the same in Float64 at an ordinary, odd size (a likelihood's gradient)
        dict(name="grad_f64_d150", kind="grad", dtype="float64", d=150, m=10_000, reps=12, qmc="Richtmyer",
             bounds="finite", cov="random"),
        # many problems of uneven dimension in one launch
        dict(name="batch_f32_d16_256", kind="batch", dtype="float32", n=256, dmin=16, dmax=256, m=2**13, reps=8,
             qmc="Sobol", bounds="finite"),
        # the sparse path at its default type
        dict(name="banded_f64_d2000", kind="banded", dtype="float64", d=2000, m=2**13, reps=12, qmc="Sobol",
             bounds="upper", rho=0.8, band=32),
        # the banded benchmark's family (bandwidth 64), forward and with gradients
        dict(name="banded_f32_d4000", kind="banded", dtype="float32", d=4000, m=2**15, reps=10, qmc="Sobol",
             bounds="upper", rho=0.9, band=64),
        dict(name="banded_grad_f32_d4000", kind="banded_grad", dtype="float32", d=4000, m=2**13, reps=10, qmc="Sobol",
             bounds="upper", rho=0.9, band=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "pass", "pass", "grad", "batch", "banded", "banded_grad"])
    dtype = rng.choice(["float64", "float32"])
    qmc = rng.choice(["Richtmyer", "Sobol"])
    bounds = rng.choice(["upper", "finite"])
    reps = rng.randint(8, 16)
    f64 = dtype == "float64"
    if kind == "batch":
        dmin = rng.randint(4, 60)
        return dict(kind=kind, dtype=dtype, n=rng.randint(20, 128 if f64 else 256), dmin=dmin,
                    dmax=rng.randint(dmin, 256), m=_log_int(rng, 1000, 2000 if f64 else 2**13), reps=8, qmc=qmc,
                    bounds=bounds)
    if kind in ("banded", "banded_grad"):
        d = _log_int(rng, 100, 2000 if f64 else 4000)
        return dict(kind=kind, dtype=dtype, d=d, m=_log_int(rng, 1000, 2**13), reps=min(reps, 10), qmc=qmc,
                    bounds=bounds, rho=round(rng.uniform(0.5, 0.95), 3), band=rng.randint(2, min(d - 1, 100)))
    if kind == "grad":
        d = _log_int(rng, 10, 400 if f64 else 1000)
        m = _log_int(rng, 1000, 10_000 if f64 else 2**15)
    else:
        d = _log_int(rng, 5, 1000)
        m = _log_int(rng, 1000, 2**14 if f64 else 2**16)
    return dict(kind=kind, dtype=dtype, d=d, m=m, reps=reps, qmc=qmc, bounds=bounds,
                cov="factor" if d >= 50 and rng.random() < 0.5 else "random")


# ---- inputs ----------------------------------------------------------------
def _correlation(S):
    s = np.sqrt(np.diag(S))
    R = S / np.outer(s, s)
    np.fill_diagonal(R, 1.0)
    return (R + R.T) / 2


def _covariance(case, d, rng):
    if case["kind"] in ("banded", "banded_grad"):
        i = np.arange(d, dtype=np.float64)
        return np.exp(np.abs(i[:, None] - i[None, :]) * math.log(case["rho"]))
    if case.get("cov") == "factor":
        B = rng.normal(0, 0.15, (d, 20))
        return _correlation(B @ B.T + np.diag(rng.uniform(0.2, 1.0, d)))
    A = rng.standard_normal((d, d + max(10, d // 2)))
    return _correlation(A @ A.T)


def _bounds(case, d, rng):
    """Around the rectangle (or orthant) that has probability 1/4 when the variables are independent."""
    if case["bounds"] == "upper":
        k = SQRT2 * float(torch.erfinv(torch.tensor(2 * 0.25 ** (1 / d) - 1, dtype=torch.float64)))
        return np.full(d, -np.inf), k * rng.uniform(0.85, 1.1, d)
    k = SQRT2 * float(torch.erfinv(torch.tensor(0.25 ** (1 / d), dtype=torch.float64)))
    return -k * rng.uniform(0.75, 1.15, d), k * rng.uniform(0.75, 1.15, d)


def _shifts(case, d, rng):
    if case["qmc"] == "Sobol":
        return rng.integers(0, 2**64, size=(d - 1, case["reps"]), dtype=np.uint64)
    sh = rng.random((d - 1, case["reps"]))
    # a Float32 problem draws its shifts in Float32
    return sh.astype(np.float32).astype(np.float64) if case["dtype"] == "float32" else sh


def _dirnums(dims):
    """Joe and Kuo's direction numbers (PyTorch's table, 30 bits), as (dims, 32) words of 32 bits."""
    V = np.zeros((dims, 32), dtype=np.uint32)
    state = torch.quasirandom.SobolEngine(dims, scramble=False).sobolstate.numpy()
    V[:, :30] = (state << 2).astype(np.uint32)
    return V


def _problems(case, seed):
    """[(Sigma, a, b, shifts)] of the case."""
    rng = np.random.default_rng(seed)
    dims = rng.integers(case["dmin"], case["dmax"] + 1, case["n"]) if case["kind"] == "batch" else [case["d"]]
    return [(_covariance(case, int(d), rng), *_bounds(case, int(d), rng), _shifts(case, int(d), rng)) for d in dims]


def prepare(case, seed):
    probs = _problems(case, seed)
    opts = D.QMC_opts(np.dtype(case["dtype"]).type, m=case["m"], max_pts=case["m"], n_reps=case["reps"])
    gen = {"qmc_type": case["qmc"]}
    if case["qmc"] == "Sobol":
        gen["sobol_dirnums"] = _dirnums(max(p[0].shape[0] for p in probs) - 1)
    st = {"kind": case["kind"], "T": np.dtype(case["dtype"]).type, "opts": opts}
    if case["kind"] == "batch":
        plan = D.BatchPlan([p[0].shape[0] for p in probs], opts, **gen)
        plan.fill([p[:3] for p in probs], [p[3] for p in probs])
        st["plan"] = plan
        return st
    S, a, b, sh = probs[0]
    gen["ushifts" if case["qmc"] == "Sobol" else "shifts"] = np.asfortranarray(sh)
    S = np.asfortranarray(S)
    if case["kind"] == "call":
        st.update(S=S, a=a, b=b, gen=gen)
        return st
    banded = case["kind"] in ("banded", "banded_grad")
    st["D"] = (D.QMCDataSparse if banded else D.QMCData)(S, a, b, opts, **gen)
    if banded:
        st["D"].truncate_band(case["band"])
    return st


def run(st):
    T = st["T"]
    if st["kind"] == "batch":
        P, err = st["plan"].run()
        return {"P": P.astype(T), "err": err.astype(T)}
    if st["kind"] in ("grad", "banded_grad"):
        if st["kind"] == "grad":
            P, err, n, da, db, G = D.qmc_pnorm_grad_sigma(st["D"])
        else:
            P, err, n, da, db, _ = D.qmc_pnorm_grad(st["D"])
        out = {"estimate": np.array([P, err], dtype=T), "n_pts": n, "da": da.astype(T), "db": db.astype(T)}
        if st["kind"] == "grad":
            out["dSigma"] = G.astype(T)
        return out
    Dat = D.QMCData(st["S"], st["a"], st["b"], st["opts"], **st["gen"]) if st["kind"] == "call" else st["D"]
    P, err, n, reps = D.qmc_pnorm(Dat, return_reps=True)
    return {"estimate": np.array([P, err], dtype=T), "n_pts": n, "reps": reps.astype(T)}


def work(case):
    """Inputs read once and outputs written once; two operations for each product of the conditioning sums (and its
    derivatives) and 50 for each normal CDF or quantile."""
    N, R = case["m"] * case["reps"], case["reps"]
    grad = case["kind"] in ("grad", "banded_grad")
    sides = 1 if case["bounds"] == "upper" else 2
    if case["kind"] == "batch":
        dims = np.random.default_rng(0).integers(case["dmin"], case["dmax"] + 1, case["n"])
    else:
        dims = np.array([case["d"]])
    by = fl = 0.0
    for d in dims.astype(float):
        terms = d * (d - 1) / 2
        if "band" in case:
            terms = min(terms, (d - 1) * case["band"])
        fl += N * (2 * terms * (3 if case["kind"] == "grad" else 2 if grad else 1)
                   + 50 * (d - 1) * (1 + sides) * (2 if grad else 1))
        if case["kind"] in ("call", "batch"):
            fl += d**3 / 3
            by += 8 * (d * d + 2 * d + (d - 1) * R)
        else:
            by += 8 * (terms + 3 * d + (d - 1) * R)
        by += 8 * (R + 2) + (8 * (2 * d + (d * d if case["kind"] == "grad" else 0)) if grad else 0)
    return {"bytes": by, "flops": fl}


# ---- the same numbers in 64 bits, plain torch --------------------------------
def _phi_erf(x):
    return 0.5 * (1.0 + torch.erf(x))


def _factor(S, a, b, pivot):
    """Correlation scaling and the Cholesky factor of many problems at once (padded with ones on the diagonal and
    infinite bounds), variables in the order of Genz's rule: the smallest remaining probability first, looked for in
    panels of 512 variables, each with its own conditional means.  -> U, a, b (in that order), order, scale."""
    P, d, _ = S.shape
    s = torch.sqrt(torch.diagonal(S, dim1=1, dim2=2))
    M = S / (s[:, :, None] * s[:, None, :])
    a, b = a / s, b / s
    if not pivot:
        return torch.linalg.cholesky(M).transpose(1, 2).contiguous(), a, b, None, s
    at, idx = torch.arange(P, device=S.device), torch.arange(d, device=S.device)
    free = torch.ones(P, d, dtype=torch.bool, device=S.device)
    rows = torch.zeros(P, d, d, dtype=S.dtype, device=S.device)
    order = idx.repeat(P, 1)  # the variable at each position; a pivot changes places with the first free one
    mean = torch.zeros_like(a)
    for i in range(d):
        if i % 512 == 0:
            mean.zero_()
            end = min(d, i + 512)
            panel = (idx >= i) & (idx < end)
        sd = torch.sqrt(torch.diagonal(M, dim1=1, dim2=2).clamp_min(0))
        lo, hi = (a - mean) / sd, (b - mean) / sd
        score = torch.erf(hi / SQRT2) - torch.erf(lo / SQRT2)
        pos = i + torch.gather(score, 1, order[:, i:end]).argmin(1)  # the first of equal ones
        k, first = order[at, pos], order[:, i].clone()
        order[at, pos], order[:, i], free[at, k] = first, k, False
        lo, hi, m = lo[at, k], hi[at, k], sd[at, k]
        y = (torch.exp(-lo * lo / 2) - torch.exp(-hi * hi / 2)) / math.sqrt(2 * math.pi) / score[at, k]
        y = torch.where(torch.isnan(y), 0.0, y * 2.0)  # score is twice the probability; padding has y = 0
        row = torch.where(free, M[at, k] / m[:, None], 0.0)
        M = M - row[:, :, None] * row[:, None, :]
        mean = mean + y[:, None] * torch.where(panel, row, 0.0)
        row[at, k] = m
        rows[:, i] = row
    U = torch.gather(rows, 2, order[:, None, :].expand(P, d, d))
    return U, torch.gather(a, 1, order), torch.gather(b, 1, order), order, s


def _sqrt_primes(n, dev):
    primes, k = [], 2
    while len(primes) < n:
        if all(k % p for p in primes if p * p <= k):
            primes.append(k)
        k += 1
    q = torch.tensor([math.sqrt(p) for p in primes], dtype=torch.float64, device=dev)
    return q - torch.floor(q)


class _Points:
    """w = |2u - 1| of QMC dimension l at the samples of points [j0, j1) of every shift, [problems, shifts * points]."""

    def __init__(self, case, shifts, d, dev):
        self.case, self.dev, m = case, dev, case["m"]
        R = case["reps"]
        if case["qmc"] == "Sobol":
            self.V = torch.from_numpy(_dirnums(d - 1).astype(np.int64)).to(dev)
            self.first = (1 << (2 * m).bit_length() - 1) + 1
            sh = np.zeros((len(shifts), d - 1, R), dtype=np.int64)
            for i, x in enumerate(shifts):
                sh[i, : x.shape[0]] = (x & np.uint64(0xFFFFFFFF)).astype(np.int64)
        else:
            self.q = _sqrt_primes(d - 1, dev)
            sh = np.zeros((len(shifts), d - 1, R))
            for i, x in enumerate(shifts):
                sh[i, : x.shape[0]] = x
        self.sh = torch.from_numpy(sh).to(dev)

    def block(self, j0, j1):
        self.j = torch.arange(j0, j1, device=self.dev)
        if self.case["qmc"] == "Sobol":
            n = self.first + self.j
            self.gray = n ^ (n >> 1)

    def w(self, l):
        sh = self.sh[:, l, :, None]
        if self.case["qmc"] == "Sobol":
            x = torch.zeros_like(self.gray)
            for bit in range(int(self.gray.max()).bit_length() if self.gray.numel() else 0):
                x = x ^ (((self.gray >> bit) & 1) * self.V[l, bit])
            u = (x ^ sh).double() * 2.0**-32
        else:
            x = (self.j + 1).double() * self.q[l]
            u = sh + (x - torch.floor(x))
            u = torch.where(u > 1, u - 1, u)
        return torch.abs(2 * u - 1).flatten(1)


def _forward(U, a, b, pts, band, keep):
    """Weights of the samples; with keep also (y, w, x_lower, x_upper, dc, free) for the reverse pass."""
    P, d = a.shape
    inv = 1 / (torch.diagonal(U, dim1=1, dim2=2) * SQRT2)
    c = _phi_erf(a[:, 0] * inv[:, 0])[:, None]
    dc = _phi_erf(b[:, 0] * inv[:, 0])[:, None] - c
    Y, kept, p = None, [], None
    eps = float(np.finfo(np.float64).eps)
    for l in range(d - 1):
        w = pts.w(l)
        if Y is None:
            Y = torch.zeros(P, d - 1, w.shape[1], dtype=torch.float64, device=w.device)
            p, dc, c = dc.expand_as(w), dc.expand_as(w), c.expand_as(w)
        v = c + w * dc
        u = v.clamp(eps, 1 - eps)
        Y[:, l] = SQRT2 * torch.erfinv(2 * u - 1)
        lo = max(0, l + 1 - band) if band else 0
        s = torch.bmm(U[:, lo:l + 1, l + 1][:, None, :], Y[:, lo:l + 1])[:, 0]
        xa, xb = (a[:, l + 1, None] - s) * inv[:, l + 1, None], (b[:, l + 1, None] - s) * inv[:, l + 1, None]
        c = _phi_erf(xa.clamp(-9, 9))
        dc = _phi_erf(xb.clamp(-9, 9)) - c
        p = p * dc
        if keep:
            kept.append((w, xa, xb, dc, (v > eps) & (v < 1 - eps)))
    return (p, Y, kept) if keep else p


def _reverse(U, a, b, p, Y, kept, dc0, band):
    """Sums over the samples of dp/da, dp/db and dp/dU (one problem)."""
    d = a.shape[0]
    rpi = 1 / math.sqrt(2 * math.pi)
    diag = torch.diagonal(U)
    ga, gb, gU = torch.zeros_like(a), torch.zeros_like(b), torch.zeros_like(U)
    sbar = torch.zeros(d, p.shape[0], dtype=torch.float64, device=p.device)
    ybar = torch.zeros_like(p)
    for t in range(d - 1, -1, -1):
        if t < d - 1:
            hi = min(d, t + 1 + band) if band else d
            ybar = U[t, t + 1:hi] @ sbar[t + 1:hi]
            w, y, ok = kept[t][0][0], Y[t], kept[t][4][0]
            ubar = torch.where(ok, ybar * torch.exp(y * y / 2) / rpi, 0.0)
        else:
            w = ubar = torch.zeros_like(p)
        if t:
            _, xa, xb, dc, _ = (x[0] for x in kept[t - 1])
            fa, fb = (torch.where(x.abs() < 9, rpi * torch.exp(-x * x), 0.0) for x in (xa, xb))
        else:
            xa, xb = (torch.full_like(p, float(x[0] / (diag[0] * SQRT2))) for x in (a, b))
            fa, fb, dc = rpi * torch.exp(-xa * xa), rpi * torch.exp(-xb * xb), torch.full_like(p, dc0)
        one = torch.where(dc > 0, p / dc, 0.0)
        da = torch.where(fa > 0, (-one + ubar * (1 - w)) * fa / diag[t], 0.0)
        db = torch.where(fb > 0, (one + ubar * w) * fb / diag[t], 0.0)
        sbar[t] = -(da + db)
        ga[t], gb[t] = da.sum(), db.sum()
        al, be = (torch.where(f > 0, x * SQRT2, 0.0) for f, x in ((fa, xa), (fb, xb)))
        gU[t, t] = -(da * al + db * be).sum()
    if not band:
        gU += torch.triu(torch.cat([Y @ sbar.T, torch.zeros(1, d, dtype=torch.float64, device=p.device)]), 1)
    return ga, gb, gU


def _sigma_gradient(S, a, b, order, ga, gb, gU):
    """Gradients in the original order and scale, through the factorisation with its order held fixed."""
    with torch.enable_grad():
        S, av, bv = (x.detach().clone().requires_grad_() for x in (S, a.nan_to_num(0, 0, 0), b.nan_to_num(0, 0, 0)))
        s = torch.sqrt(torch.diagonal(S))
        U = torch.linalg.cholesky((S / (s[:, None] * s[None, :]))[order][:, order]).T
        f = (U * gU).sum() + (((av / s)[order]) * ga).sum() + (((bv / s)[order]) * gb).sum()
        f.backward()
    return av.grad, bv.grad, (S.grad + S.grad.T) / 2


def exact(case, seed):
    if work(case)["flops"] > 4e12:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    probs = _problems(case, seed)
    n, d, m, R = len(probs), max(p[0].shape[0] for p in probs), case["m"], case["reps"]
    S = torch.eye(d, dtype=torch.float64).repeat(n, 1, 1)
    a, b = torch.full((n, d), -torch.inf, dtype=torch.float64), torch.full((n, d), torch.inf, dtype=torch.float64)
    for i, (Si, ai, bi, _) in enumerate(probs):
        k = ai.shape[0]
        S[i, :k, :k], a[i, :k], b[i, :k] = torch.from_numpy(Si), torch.from_numpy(ai), torch.from_numpy(bi)
    S, a, b = S.to(dev), a.to(dev), b.to(dev)
    band, grad = case.get("band", 0), case["kind"] in ("grad", "banded_grad")
    U, au, bu, order, s = _factor(S, a, b, not band)
    if band:
        U = torch.triu(U) - torch.triu(U, band + 1)
    pts = _Points(case, [p[3] for p in probs], d, dev)
    per = max(1, min(m, int((4e9 if grad else 1.2e10) // (8 * n * d * R * (6 if grad else 1)))))
    total, g = torch.zeros(n, R, dtype=torch.float64, device=dev), [0.0, 0.0, 0.0]
    dc0 = float((_phi_erf(bu[0, 0] / (U[0, 0, 0] * SQRT2)) - _phi_erf(au[0, 0] / (U[0, 0, 0] * SQRT2))))
    for j0 in range(0, m, per):
        pts.block(j0, min(m, j0 + per))
        if grad:
            p, Y, kept = _forward(U, au, bu, pts, band, True)
            g = [x + y for x, y in zip(g, _reverse(U[0], au[0], bu[0], p[0], Y[0], kept, dc0, band))]
            del Y, kept
        else:
            p = _forward(U, au, bu, pts, band, False)
        total += p.reshape(n, R, -1).sum(2)
    reps = total / m
    P = reps.mean(1)
    err = 3 * torch.sqrt(((reps - P[:, None]) ** 2).mean(1) / (R - 1))
    P, err, reps = P.cpu().numpy(), err.cpu().numpy(), reps.cpu().numpy()
    if case["kind"] == "batch":
        return {"P": P, "err": err}
    out = {"estimate": np.array([P[0], err[0]]), "n_pts": None}
    if not grad:
        out["reps"] = reps[0]
        return out
    ga, gb, gU = (x / (m * R) for x in g)
    if band:
        da, db = ga / s[0], gb / s[0]
    else:
        da, db, G = _sigma_gradient(S[0], a[0], b[0], order[0], ga, gb, gU)
        out["dSigma"] = G.cpu().numpy()
    out["da"], out["db"] = da.cpu().numpy(), db.cpu().numpy()
    return out
