"""Infinite and undefined values: what they touched before the loops over pairs
lost their branches, and nothing else.  A Lambert coefficient exp(a) that
overflows makes a point's brightness infinite if it sees a facet and leaves it
zero if it sees none (opposite Sun and Earth); a point whose time is not a number
sees none."""
import numpy as np
import pytest

from test_gpu_adjoint_curves import _desc

pytestmark = pytest.mark.gpu

DARK, LOST = 7, 40  # a point opposite the Sun; one without a time
N = 150


def _problem(lmax, nrows, lost, **more):
    d = _desc(11, [(0, N)], lmax, nrows, False)
    d["ee0"][DARK] = -d["ee"][DARK]
    if lost:
        d["tim"][LOST] = np.nan
    return dict(d, **more)


def _open(native, form, desc):
    g = native.PeriodSearch(desc=desc, form={"fp64": native.PS_FORM_FP64, "fast": native.PS_FORM_FAST}[form])
    g.set_conw_r(0.4)
    return g, np.concatenate([g.array("cg_first"), [0.4, 1.0, 24 * 2 * np.pi * g.freq_start, 0.5, 0.1, -0.5, np.log(0.1), 1.0]])


# coefficient counts with and without the column on the FP64 pipe
@pytest.mark.parametrize("form", ["fp64", "fast"])
@pytest.mark.parametrize("lmax,nrows", [(1, 3), (2, 4), (4, 5), (8, 9)])
def test_rows(native, form, lmax, nrows):
    g, a = _open(native, form, _problem(lmax, nrows, True))
    C = g.ncoef
    seen = np.ones(N, bool)
    seen[[DARK, LOST]] = False
    y, J = g.model(a)
    assert np.all(np.isfinite(y)) and np.all(y[:N][seen] > 0) and np.all(y[:N][~seen] == 0)
    assert np.all(np.isfinite(J[:N][seen])) and np.all(np.isfinite(J[DARK]))
    for log_cl, cls in ((800.0, 1.0), (-2.0, np.inf), (705.0, 1e308)):
        a[C + 6], a[C + 7] = log_cl, cls
        y, J = g.model(a)
        assert np.all(np.isposinf(y[:N][seen])) and np.all(y[:N][~seen] == 0), (log_cl, cls)
        assert np.all(np.isposinf(J[:N][seen, 0])) and np.all(J[:N][~seen, :C] == 0), (log_cl, cls)
    g.close()


def test_fit_with_a_point_without_time(native):
    """The point is dark in the model of every trial, as in the Jacobian's: the fit
    takes steps, and its chi2 is the evaluation's at its parameters."""
    d = _problem(3, 6, True, stop_condition=12.0)
    g, _ = _open(native, "fp64", d)
    for pole in (2, 7):
        r, cg = g.fit(g.freq_start, pole, params=True)
        assert r["niter"] == 12 and r["status"] == 0
        assert np.isfinite(r["chisq"]) and r["chisq"] == g.mrqcof(cg)[2]
        assert not np.array_equal(cg[:g.ncoef], g.array("cg_first"))  # some step was accepted
    g.close()


@pytest.mark.parametrize("lmax,nrows", [(2, 4), (5, 7)])
def test_matrix_free_calls(native, lmax, nrows):
    """chi2, beta and products as the explicit evaluation has them: infinite where
    the model is, finite in the shape columns where a point without a time is dark
    (its rotation columns are not numbers in fused arithmetic)."""
    d = _problem(lmax, nrows, True)
    g, a = _open(native, "fast", d)
    e, _ = _open(native, "fp64", d)
    C, v = g.ncoef, np.ones(g.mfit)
    alpha, beta, x2 = e.mrqcof(a)
    x2_g, beta_g = g.chi2_grad(a)
    assert abs(x2_g - x2) <= 1e-10 * x2
    assert np.all(np.abs(beta_g - beta)[:C] <= 1e-10 * np.sqrt(np.diag(alpha) * x2)[:C])
    for log_cl in (800.0, 705.0):
        a[C + 6], a[C + 7] = log_cl, 1e308
        x2_g, beta_g = g.chi2_grad(a)
        assert np.isposinf(x2_g) and e.mrqcof(a)[2] == x2_g
        assert not np.any(np.isfinite(beta_g[:C]))
    g.close()
    # an infinite weight: no finite chi2; an infinite brightness where no facet is
    # seen: no facet's sum takes part in it
    d = _problem(lmax, nrows, False)
    d["weight"][DARK] = np.inf
    g, a = _open(native, "fast", d)
    assert not np.isfinite(g.chi2_grad(a)[0])
    g.close()
    d = _problem(lmax, nrows, False)
    d["brightness"][DARK] = np.inf
    g, a = _open(native, "fast", d)
    x2_g, beta_g = g.chi2_grad(a)
    assert np.isposinf(x2_g) and np.all(np.isfinite(beta_g[1:C]))
    g.close()


@pytest.mark.parametrize("seed,lmax,nrows,poles", [(3, 3, 6, (6, 7)), (21, 1, 4, (5, 10))])
def test_fits_that_run_into_overflow(native, seed, lmax, nrows, poles):
    """Relative lightcurves alone do not determine the Lambert coefficient: these
    fits run to exp(355) and more, where y sum(dy) overflows in the normalisation,
    and freeze with a matrix of NaNs (status 1).  The Jacobian-free fit does too."""
    d = _desc(2000 + seed, [(1, 40), (1, 30)], lmax, nrows, False)
    d.update(stop_condition=6.0, per_start=7.9, per_end=8.1, weight=np.ones(70))
    g, _ = _open(native, "fp64", d)
    f, _ = _open(native, "fast", d)
    for pole in poles:
        r, cg = g.fit(g.freq_start, pole, params=True)
        assert r["status"] == 1 and cg[g.ncoef + 6] > 355
        j = f.fit_jfree(g.freq_start, pole)
        assert j["status"] == 1 and j["niter"] == r["niter"]
        assert abs(j["chisq"] - r["chisq"]) <= 1e-9 * r["chisq"]
        assert not np.any(np.isfinite(f.gn_product(cg, np.ones(f.mfit))))
    g.close()
    f.close()
