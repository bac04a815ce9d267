"""Performance cases of the period scan: the calls a program makes, each
through its public entry point (`PeriodSearch`, `PeriodSearchBatch`).

Sizes are the ones the tests, goldens and the benchmark use: survey photometry
(about 120 calibrated points, lmax 3, 6 rows = 288 facets), dense data (500
points in six nights and a sparse set, lmax 3), the production sparse search
(760 points, lmax 6, 10 rows = 800 facets), uneven batches (100 to 5000
points, lmax 6) and the large shape (20 000 points, lmax 8, 16 rows = 2048
facets).  Inputs are synthetic lightcurves of a seeded convex body with
noise; dense nights are relative, sparse sets calibrated.

Scans and fits in the reference-order form run the production stop rule, 50
steps per fit.  LM paths amplify rounding by about a factor of three every two
steps once they crawl along flat valleys, so the forms that differ from the
reference order by rounding are run under the stop rules of a first, coarse
pass (8 to 12 steps, or an rms improvement under 1e-2), where a scan of the
same periods is reproducible to about 1e-10.  The work of a step is the same.
"""
import math

import numpy as np
import torch

import periodsearch_b200 as ps

FORMS = {"fp64": ps.PS_FORM_FP64, "fast": ps.PS_FORM_FAST}


def listed():
    survey = dict(nights=0, per_night=0, sparse=118, lmax=3, rows=6)
    dense = dict(nights=6, per_night=50, sparse=200, lmax=3, rows=6)
    sparse = dict(nights=2, per_night=80, sparse=600, lmax=6, rows=10)
    large = dict(nights=40, per_night=100, sparse=16000, lmax=8, rows=16)
    return [
        # one fit of survey photometry in the default form: the smallest call
        dict(name="fit_survey_fp64", call="fit", form="fp64", steps=50, **survey),
        # one fit of the production shape, to refine one candidate period
        dict(name="fit_sparse_fast", call="fit", form="fast", steps=12, **sparse),
        # model rows and Jacobian at given parameters, for residual plots
        dict(name="model_dense_fp64", call="model", form="fp64", steps=50, **dense),
        # chi2 and its gradient, one call of an outer optimiser
        dict(name="grad_sparse", call="grad", form="fast", steps=50, **sparse),
        # Gauss-Newton product at the large shape
        dict(name="gn_large", call="gn", form="fast", steps=50, **large),
        # a short scan of survey photometry (fewer fits than the GPU has slots)
        dict(name="scan_survey_fp64", call="scan", form="fp64", steps=50, periods=20, **survey),
        # the production search in the drop-in form, 600 fits
        dict(name="scan_sparse_fp64", call="scan", form="fp64", steps=50, periods=60, **sparse),
        # the production search in the fast form, 2400 fits of a coarse pass
        dict(name="scan_sparse_fast", call="scan", form="fast", steps=10, periods=240, **sparse),
        # many asteroids of uneven size in one launch, fits stopped by convergence
        dict(name="batch_fast", call="batch", form="fast", steps=0, asteroids=32, periods=4, n_min=100, n_max=5000,
             lmax=6, rows=10),
        # the large shape, one fit per SM
        dict(name="scan_large_fast", call="scan", form="fast", steps=8, periods=14, **large),
        # a whole work unit as the application runs it: the convexity pre-pass,
        # then the scan
        dict(name="unit_dense_fp64", call="unit", form="fp64", steps=50, periods=40, **dense),
        # a Jacobian-free fit of the large shape
        dict(name="jfree_large", call="jfree", form="fast", steps=8, **large),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more call: any of the listed kinds, sizes spread over the ranges
    they stand for, mostly not multiples of anything."""
    call = rng.choice(["fit", "model", "grad", "gn", "scan", "scan", "scan", "batch", "unit", "jfree"])
    lmax = rng.choice([2, 3, 4, 5, 6, 6, 7, 8])
    rows = rng.randint(max(3, lmax), min(16, lmax + 6))
    n = _log(rng, 60, 6000)
    nights = rng.randint(0, 8)
    per_night = max(10, int(n * rng.uniform(0.1, 0.6)) // max(nights, 1)) if nights else 0
    shape = dict(nights=nights, per_night=per_night, sparse=max(40, n - nights * per_night), lmax=lmax, rows=rows)
    size = (nights * per_night + shape["sparse"]) * 8 * rows * rows * (30 + (lmax + 1) ** 2)
    big = 760 * 800 * 79  # the production shape
    if call == "batch":
        return dict(call="batch", form="fast", steps=0, asteroids=rng.randint(3, 24), periods=rng.randint(1, 4),
                    n_min=100, n_max=rng.randint(600, 4000), lmax=min(lmax, 6), rows=min(rows, 10))
    if call == "grad" or call == "gn":
        return dict(call=call, form="fast", steps=50, **shape)
    if call == "jfree":
        return dict(call=call, form="fast", steps=rng.randint(6, 9), **shape)
    form = rng.choice(["fp64", "fast"])
    if call == "unit":
        form = "fp64"
    if call == "model":
        return dict(call=call, form=form, steps=50, **shape)
    if call == "fit":
        return dict(call=call, form=form, steps=50 if form == "fp64" and size < big else rng.randint(6, 11), **shape)
    steps = 50 if form == "fp64" and size < 2 * big else rng.randint(6, 10)
    most = 0.5 * 2400 * 10 * big / (size * steps) * (0.4 if form == "fp64" else 1.0) / 10
    periods = max(2, min(400, _log(rng, 2, max(3, int(most)))))
    return dict(call=call, form=form, steps=steps, periods=periods, **shape)


# ---- inputs -----------------------------------------------------------------


def _unit(v):
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _orbit(radius, days, incl, phase, t):
    a = phase + 2 * math.pi * t / days
    x, y = radius * np.cos(a), radius * np.sin(a)
    return np.stack([x, y * math.cos(incl), y * math.sin(incl)], axis=1)


def _spin(beta_p, lam):
    cb, sb, cl, sl = math.cos(beta_p), math.sin(beta_p), math.cos(lam), math.sin(lam)
    return np.array([[cb * cl, cb * sl, -sb], [-sl, cl, 0.0], [sb * cl, sb * sl, cb]])


def _lightcurves(shape, seed, stop, stop_min, periods):
    """A seeded convex body's lightcurves as the arrays PeriodSearch(desc=...)
    takes: an ellipsoid with bumps under Lambert + Lommel-Seeliger scattering,
    observed from the Earth over eight years, 3 % noise."""
    g = np.random.default_rng(seed)
    k = np.arange(400) + 0.5
    z = 1 - 2 * k / 400
    az = math.pi * (1 + 5**0.5) * k
    r = np.sqrt(1 - z * z)
    nor = np.stack([r * np.cos(az), r * np.sin(az), z], axis=1)
    ax = np.array([1.0, g.uniform(0.6, 0.9), g.uniform(0.4, 0.7)])
    area = np.prod(ax) ** 2 / np.sum((ax * nor) ** 2, axis=1) ** 2
    area *= np.exp(0.15 * np.sin(nor @ g.normal(0, 2.5, (3, 3)) + g.uniform(0, 6, 3)).sum(axis=1))
    area *= 4 * math.pi / 400
    lam, beta, hours = g.uniform(0, 2 * math.pi), g.uniform(-1.4, 1.4), g.uniform(4, 12)
    span, ph_a, ph_e = 8 * 365.25, g.uniform(0, 6), g.uniform(0, 6)
    ast = lambda t: _orbit(2.5, 365.25 * 2.5**1.5, 0.14, ph_a, t)  # noqa: E731
    earth = lambda t: _orbit(1.0, 365.25, 0.0, ph_e, t)  # noqa: E731

    def epochs(n):
        got = np.zeros(0)
        while got.size < n:
            t = g.uniform(0, span, 4 * n + 16)
            to_a, to_s = ast(t) - earth(t), -earth(t)
            c = np.sum(to_a * to_s, 1) / np.linalg.norm(to_a, axis=1) / np.linalg.norm(to_s, axis=1)
            got = np.concatenate([got, t[c < 0.5]])
        return np.sort(got[:n])

    curves = [(1, np.sort(t0 + g.uniform(0, 0.33, shape["per_night"]))) for t0 in epochs(shape["nights"])]
    curves.append((0, epochs(shape["sparse"])))
    t = np.concatenate([c[1] for c in curves])
    sun, obs = _unit(-ast(t)), _unit(earth(t) - ast(t))
    f = np.fmod(24 * 2 * math.pi / hours * t, 2 * math.pi)
    rot = _spin(math.pi / 2 - beta, lam)

    def body(v):
        w = v @ rot.T
        return np.stack([np.cos(f) * w[:, 0] + np.sin(f) * w[:, 1], np.cos(f) * w[:, 1] - np.sin(f) * w[:, 0], w[:, 2]], 1)

    mu, mu0 = body(obs) @ nor.T, body(sun) @ nor.T
    see = (mu > 1e-8) & (mu0 > 1e-8)
    s = np.where(see, mu * mu0 * (0.1 + 1 / np.where(see, mu + mu0, 1.0)), 0.0)
    alpha = np.arccos(np.clip(np.sum(sun * obs, 1), -1, 1))
    bright = (1 + 0.5 * np.exp(-alpha / 0.1) - 0.5 * alpha) * (s @ area) * (1 + 0.03 * g.standard_normal(t.size))
    # as the application prepares a work unit: per-lightcurve mean brightness as
    # sigma, the size scale from the lowest phase angle of the calibrated sets
    sig = np.empty(t.size)
    at, first = 0, None
    for rel, c in curves:
        sig[at : at + c.size] = bright[at : at + c.size].mean()
        if not rel and (first is None or alpha[at] < alpha[first]):
            first = at
        at += c.size
    fit = math.sqrt(2 * sig[first] / (0.5 * math.pi * (1 + math.cos(alpha[first]))))
    escl = 0.8 * fit / math.sqrt((1.05 + 0.95 + 1.05 * 0.95) / 3)
    jd_min, jd_max = float(t.min()), float(t.max())
    step = 0.5 / (jd_max - jd_min) / 24 * 0.5
    half = (periods + 4) / 2
    return dict(
        lc_points=[c.size for _, c in curves], lc_relative=[rel for rel, _ in curves], tim=t, ee=obs, ee0=sun,
        brightness=bright, sig=sig, weight=np.ones(t.size), per_start=1 / (1 / hours + half * step), per_step_coef=0.5,
        per_end=1 / (1 / hours - half * step), ia_prd=1, phi0_rad=0.0, conw=0.1, lmax=shape["lmax"],
        mmax=shape["lmax"], nrows=shape["rows"], par=[0.5, 0.1, -0.5], ia_par=[1, 1, 1], cl=0.1, ia_cl=0,
        stop_condition=stop, n_iter_min=stop_min, alamda_incr=5.0, alamda_start=0.1, jd_min=jd_min, jd_max=jd_max,
        escl=escl), 1 / hours


def _desc(case, seed):
    return _lightcurves(case, seed, float(case["steps"]), 5, case.get("periods", 1))


CONVEXITY = 3.2  # convexity weight times escl^2 that the pre-pass usually ends at


def _params(case, seed, desc, freq):
    """Parameters and a direction as an outer optimiser has them: the starting
    ellipsoid with small changes, a pole, the trial rotation rate."""
    g = np.random.default_rng(seed + 77)
    c = (case["lmax"] + 1) ** 2
    cg = _ellipsoid(_facets(case["rows"]), case["lmax"], desc["escl"])
    a = np.concatenate([cg, [g.uniform(0.5, 2.5), g.uniform(0, 6), 2 * math.pi * 24 * freq, 0.5, 0.1, -0.5, math.log(0.1), 1.0]])
    size = _legendre(_facets(case["rows"]), case["lmax"]).max(axis=0)
    a[:c] += g.normal(0, 0.03, c) / size
    v = g.normal(0, 1, c + 6) / np.concatenate([size, [1, 1, 10, 1, 1, 1]])
    return a, v


def prepare(case, seed):
    if case["call"] == "batch":
        g = np.random.default_rng(seed)
        ctxs = []
        for i in range(case["asteroids"]):
            n = int(round(math.exp(g.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
            nights = int(g.integers(0, 1 + n // 80))
            shape = dict(nights=nights, per_night=int(g.integers(30, 60)) if nights else 0, lmax=case["lmax"],
                         rows=case["rows"], sparse=0)
            shape["sparse"] = max(40, n - nights * shape["per_night"])
            desc, _ = _lightcurves(shape, seed * 1000 + i, 1e-2, 5, case["periods"])
            ctxs.append(_open(desc, "fast"))
        one = np.ones(len(ctxs), dtype=np.int32)
        return dict(case=case, ctxs=ctxs, batch=ps.PeriodSearchBatch(ctxs), first=one, last=case["periods"] * one)
    desc, freq = _desc(case, seed)
    state = dict(case=case, ctx=_open(desc, case["form"]), freq=freq, start=desc["conw"] / desc["escl"] ** 2)
    if case["call"] in ("model", "grad", "gn"):
        state["a"], state["v"] = _params(case, seed, desc, freq)
    return state


def _open(desc, form):
    ctx = ps.PeriodSearch(desc=desc, form=FORMS[form])
    ctx.set_conw_r(CONVEXITY / desc["escl"] ** 2)
    return ctx


def _columns(records):
    return {k: np.ascontiguousarray(records[k]) for k in ps.RECORD_DTYPE.names}


def _fit_out(rec, cg):
    return dict(params=cg, rms=float(rec["dev"]), chi2=float(rec["chisq"]), area=float(rec["totarea"]),
                steps=int(rec["niter"]), status=int(rec["status"]))


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "batch":
        return _columns(np.concatenate(state["batch"].scan(state["first"], state["last"])))
    ctx = state["ctx"]
    if call == "fit":
        return _fit_out(*ctx.fit(state["freq"], 5, params=True))
    if call == "jfree":
        return _fit_out(*ctx.fit_jfree(state["freq"], 5, params=True))
    if call == "model":
        y, jac = ctx.model(state["a"])
        return dict(y=y, jac=jac)
    if call == "grad":
        chi2, beta = ctx.chi2_grad(state["a"])
        return dict(chi2=chi2, beta=beta)
    if call == "gn":
        return ctx.gn_product(state["a"], state["v"])
    if call == "scan":
        return _columns(ctx.scan(1, case["periods"]))
    # a work unit: the pre-pass from the input's convexity weight, then the scan
    ctx.set_conw_r(state["start"])
    conw_r = ctx.precalc()
    return dict(_columns(ctx.scan(1, case["periods"])), conw_r=conw_r)


def work(case):
    """Operations: per (point, facet) pair the two cosines (10), the
    visibility tests, and for the visible ones (45 %) the scattering terms
    (about 40 with derivatives, 10 without); the shape block of the Jacobian
    as a plain product (2 per pair and coefficient) where a call has one, and
    the normal matrix (mfit^2 per row).  A fit of s steps evaluates the model
    s times and the Jacobian at about half its steps.  Bytes: the point table
    and the outputs."""
    c = (case["lmax"] + 1) ** 2
    facets = 8 * case["rows"] ** 2
    mfit, ma = c + 6, c + 8
    if case["call"] == "batch":
        span = case["n_max"] - case["n_min"]
        n = case["asteroids"] * span / math.log(case["n_max"] / case["n_min"])
        fits, steps = 10 * case["periods"], 12
    else:
        n = case["nights"] * case["per_night"] + case["sparse"]
        fits = {"scan": 10 * case.get("periods", 0), "unit": 10 * case.get("periods", 0) + 100}.get(case["call"], 1)
        steps = case["steps"]
    pairs = n * facets
    full = pairs * (10 + 0.45 * 40 + 2 * c) + n * mfit * (mfit + 1)
    model = pairs * (10 + 0.45 * 10)
    table = 12 * 8 * n
    if case["call"] == "model":
        return {"bytes": table + 8 * n * (ma + 1), "flops": full}
    if case["call"] in ("grad", "gn"):
        return {"bytes": table + 8 * facets * c, "flops": pairs * (2 * 10 + 0.45 * 60) + 4 * facets * c}
    return {"bytes": table + 48 * fits / 10 + 8 * facets * c, "flops": fits * steps * (model + 0.5 * full)}


# ---- the same in 64 bits, without the framework -----------------------------


def _facets(rows):
    """Normals and areas of the triangulated sphere: `rows` rings of triangles
    per octant, ring i with 4 i nodes."""
    ring = [[(0.0, 0.0)]]
    for i in range(1, 2 * rows):
        m = min(i, 2 * rows - i)
        ring.append([(i * math.pi / (2 * rows), j * math.pi / (2 * m)) for j in range(4 * m)])
    ring.append([(math.pi, 0.0)])
    tri = []
    for i in range(1, rows + 1):  # between ring i - 1 and ring i, and mirrored
        for o in range(4):
            for j in range(i):
                lo = lambda q: (i, (o * i + q) % (4 * i))  # noqa: E731
                up = lambda q: (i - 1, (o * (i - 1) + q) % max(1, 4 * (i - 1)))  # noqa: E731
                new = [(lo(j), lo(j + 1), up(j))]
                if j:
                    new.append((up(j - 1), lo(j), up(j)))
                tri += new + [tuple((2 * rows - r, q) for r, q in t) for t in new]
    xyz = lambda v: (math.sin(v[0]) * math.cos(v[1]), math.sin(v[0]) * math.sin(v[1]), math.cos(v[0]))  # noqa: E731
    p = np.array([[xyz(ring[r][q]) for r, q in t] for t in tri])
    n = np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    n *= np.sign(np.sum(n * p[:, 0], axis=1))[:, None]
    size = np.linalg.norm(n, axis=1)
    return n / size[:, None], 0.5 * size


def _columns_of(lmax):
    for m in range(lmax + 1):
        for l in range(m, lmax + 1):  # noqa: E741
            yield l, m, 0
            if m:
                yield l, m, 1


def _legendre(grid, lmax):
    """|P_lm| of the facet normals, a column per shape coefficient."""
    x = grid[0][:, 2]
    s = np.sqrt(1 - x * x)
    p = {}
    for m in range(lmax + 1):
        p[m, m] = np.prod(np.arange(1, 2 * m, 2, dtype=float)) * s**m if m else np.ones_like(x)
        for l in range(m + 1, lmax + 1):  # noqa: E741
            p[l, m] = ((2 * l - 1) * x * p[l - 1, m] - ((l + m - 1) * p[l - 2, m] if l - 2 >= m else 0)) / (l - m)
    return np.stack([p[l, m] for l, m, _ in _columns_of(lmax)], axis=1)


def _basis(grid, lmax):
    az = np.arctan2(grid[0][:, 1], grid[0][:, 0])
    trig = np.stack([np.sin(m * az) if odd else np.cos(m * az) for _, m, odd in _columns_of(lmax)], axis=1)
    return _legendre(grid, lmax) * trig


def _ellipsoid(grid, lmax, escl):
    a, b, c = 1.05 * escl, 1.00 * escl, 0.95 * escl
    n = grid[0]
    rhs = 2 * (math.log(a * b * c) - np.log((a * n[:, 0]) ** 2 + (b * n[:, 1]) ** 2 + (c * n[:, 2]) ** 2))
    m = _basis(grid, lmax)
    size = np.linalg.norm(m, axis=0)
    return np.linalg.lstsq(m / size, rhs, rcond=None)[0] / size


class _Model:
    """The model, its Jacobian and the LM loop in plain torch, 64 bits."""

    def __init__(self, desc, conw_r):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t64 = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=dev)  # noqa: E731
        grid = _facets(desc["nrows"])
        self.nor, self.darea, self.basis = t64(grid[0]), t64(grid[1]), t64(_basis(grid, desc["lmax"]))
        self.t, self.e, self.e0 = t64(desc["tim"]), t64(desc["ee"]), t64(desc["ee0"])
        self.alpha = torch.acos((self.e * self.e0).sum(1))
        three = [1.0] * 3
        self.obs = t64(np.concatenate([desc["brightness"], [0.0] * 3]))
        self.w = t64(np.concatenate([1 / desc["sig"] ** 2, [conw_r**2] * 3]))
        self.sig, self.conw_r, self.n = t64(np.concatenate([desc["sig"], three])), conw_r, len(desc["tim"])
        self.curves, at = [], 0
        for k, rel in zip(desc["lc_points"], desc["lc_relative"]):
            self.curves.append((rel, at, at + k))
            at += k
        c = self.basis.shape[1]
        self.free = list(range(c + 6))  # scattering coefficients fixed
        if all(desc["lc_relative"]):
            self.free.remove(0)
        self.dev = dev

    def rows(self, a):
        c = self.basis.shape[1]
        x = torch.as_tensor(a, dtype=torch.float64, device=self.dev)
        area = self.darea * torch.exp(self.basis @ x[:c])
        cl, cls, om = math.exp(a[c + 6]), a[c + 7], a[c + 2]
        b, l = a[c], a[c + 1]  # noqa: E741
        cb, sb, co, si = math.cos(b), math.sin(b), math.cos(l), math.sin(l)
        mats = [[[cb * co, cb * si, -sb], [-si, co, 0], [sb * co, sb * si, cb]],
                [[-sb * co, -sb * si, -cb], [0, 0, 0], [cb * co, cb * si, -sb]],
                [[-cb * si, cb * co, 0], [-co, -si, 0], [-sb * si, sb * co, 0]]]
        mats = [torch.tensor(m, dtype=torch.float64, device=self.dev) for m in mats]
        y = torch.empty(self.n + 3, dtype=torch.float64, device=self.dev)
        jac = torch.zeros(self.n + 3, c + 8, dtype=torch.float64, device=self.dev)
        for i in range(0, self.n, 2048):
            k = slice(i, min(self.n, i + 2048))
            f = torch.fmod(om * self.t[k], 2 * math.pi)
            cf, sf, t, zero = torch.cos(f), torch.sin(f), self.t[k], torch.zeros_like(f)
            turn = lambda v: torch.stack([cf * v[:, 0] + sf * v[:, 1], cf * v[:, 1] - sf * v[:, 0], v[:, 2]], 1)  # noqa: E731,B023
            dturn = lambda v: torch.stack([t * (cf * v[:, 1] - sf * v[:, 0]), -t * (cf * v[:, 0] + sf * v[:, 1]), zero], 1)  # noqa: E731,B023
            e = [turn(self.e[k] @ m.T) for m in mats] + [dturn(self.e[k] @ mats[0].T)]
            e0 = [turn(self.e0[k] @ m.T) for m in mats] + [dturn(self.e0[k] @ mats[0].T)]
            mu, mu0 = e[0] @ self.nor.T, e0[0] @ self.nor.T
            see = (mu > 1e-8) & (mu0 > 1e-8)
            d = torch.where(see, mu + mu0, torch.ones_like(mu))
            s = torch.where(see, mu * mu0 * (cl + cls / d), torch.zeros_like(mu))
            ds = torch.where(see, cls * (mu0 / d) ** 2 + cl * mu0, torch.zeros_like(mu))
            ds0 = torch.where(see, cls * (mu / d) ** 2 + cl * mu, torch.zeros_like(mu))
            ex = torch.exp(-self.alpha[k] / a[c + 4])
            sc = 1 + a[c + 3] * ex + a[c + 5] * self.alpha[k]
            br = s @ area
            y[k] = br * sc
            jac[k, :c] = sc[:, None] * ((s * area) @ self.basis)
            for q in range(3):
                dm, dm0 = e[q + 1] @ self.nor.T, e0[q + 1] @ self.nor.T
                jac[k, c + q] = sc * ((ds * dm + ds0 * dm0) @ area)
            jac[k, c + 3] = br * ex
            jac[k, c + 4] = br * a[c + 3] * ex * self.alpha[k] / a[c + 4] ** 2
            jac[k, c + 5] = br * self.alpha[k]
            both = torch.where(see, mu * mu0, torch.zeros_like(mu))
            jac[k, c + 6] = sc * (both @ area) * cl
            jac[k, c + 7] = sc * ((both / d) @ area)
        y[self.n :] = self.nor.T @ area
        jac[self.n :, :c] = (self.nor * area[:, None]).T @ self.basis
        for rel, i, j in self.curves:
            if rel:
                ave = y[i:j].sum()
                coef = (self.sig[i:j] * (j - i) / ave)[:, None]
                jac[i:j] = coef * (jac[i:j] - y[i:j, None] * jac[i:j].sum(0) / ave)
                y[i:j] = coef[:, 0] * y[i:j]
                jac[i:j, 0] = 0
        self.chk, self.area = y[self.n :].clone(), area.sum()
        return y, jac

    def normal(self, a):
        y, jac = self.rows(a)
        dy, jf = self.obs - y, jac[:, self.free]
        return (jf * self.w[:, None]).T @ jf, jf.T @ (self.w * dy), float((self.w * dy * dy).sum())

    def fit(self, a, steps, grow, lam):
        """The LM loop with a fixed number of steps."""
        alpha, beta, best = self.normal(a)
        chk, area = self.chk, self.area
        for _ in range(steps):
            da = torch.linalg.solve(alpha + lam * torch.diag(torch.diagonal(alpha)), beta).cpu().numpy()
            trial = a.copy()
            trial[self.free] += da
            al, be, chi2 = self.normal(trial)
            if chi2 < best:
                a, alpha, beta, best, chk, area, lam = trial, al, be, chi2, self.chk, self.area, lam / grow
            else:
                lam *= grow
        r = best - float((chk * chk).sum()) * self.conw_r**2
        return dict(params=a, rms=math.sqrt(r / self.n), chi2=best, area=None, steps=None, status=None)


def exact(case, seed):
    call = case["call"]
    if call in ("scan", "unit", "batch") or call in ("fit", "jfree") and case["steps"] > 12:
        return None  # hundreds of fits, or a path too long to be determined in 64 bits
    desc, freq = _desc(case, seed)
    model = _Model(desc, CONVEXITY / desc["escl"] ** 2)
    a, v = _params(case, seed, desc, freq)
    if call == "model":
        y, jac = model.rows(a)
        return dict(y=y, jac=jac)
    if call == "grad":
        _, beta, chi2 = model.normal(a)
        return dict(chi2=chi2, beta=beta)
    if call == "gn":
        _, jac = model.rows(a)
        jf = jac[:, model.free]
        return (jf.T @ (model.w * (jf @ torch.as_tensor(v, device=model.dev)))).cpu()
    c = (case["lmax"] + 1) ** 2
    a[:c] = _ellipsoid(_facets(case["rows"]), case["lmax"], desc["escl"])
    a[c], a[c + 1] = math.radians(90 - 60), math.radians(60)  # the fifth starting pole
    return model.fit(a, case["steps"], desc["alamda_incr"], desc["alamda_start"])
