"""The model pass takes four facets at a time, without branches, and (in the
reference-order form) divides through one reciprocal per pair: the trial points
of a fit must still follow the oracle's path.  Sizes at the edges: 8 nrows^2
facets around the staged chunk of 128 and its blocks of four, point counts
around a warp, a block of 256 threads and the four points a thread takes."""
import numpy as np
import pytest

from conftest import golden_path
from periodsearch_b200 import synth

pytestmark = pytest.mark.gpu

FIT_TOL = 1e-9  # the fits' bar against the oracle


@pytest.mark.parametrize("form", ["fp64", "fast"])
@pytest.mark.parametrize("nrows,points", [(1, 31), (3, 33), (4, 255), (5, 257), (4, 1030)])
def test_short_fits_follow_the_oracle(native, oracle_lib, tmp_path, form, nrows, points):
    w = synth.make_workload("model_pass", 40 + nrows, dense_lcs=0, dense_pts=0, sparse_pts=points, years=6, true_lmax=2,
                            fit_lmax=1 if nrows == 1 else 2, nrows=nrows, noise=0.02, n_periods=2, stop_condition=8)
    path = synth.write_input(w, str(tmp_path))
    o = oracle_lib.Oracle(path)
    o.set_conw_r(o.conw_r)
    g = native.PeriodSearch(path, form={"fp64": native.PS_FORM_FP64, "fast": native.PS_FORM_FAST}[form])
    g.set_conw_r(o.conw_r)
    for pole in (2, 9):
        ro, cg_o = o.fit(o.freq(1), pole)
        rg, cg = g.fit(o.freq(1), pole, params=True)
        assert rg["niter"] == int(ro["niter"]) and rg["status"] == int(ro["status"])
        assert abs(rg["chisq"] - ro["chisq"]) <= FIT_TOL * abs(ro["chisq"])
        assert abs(rg["totarea"] - ro["totarea"]) <= FIT_TOL * abs(ro["totarea"])
        assert abs(rg["dark"] - ro["dark"]) <= FIT_TOL * max(abs(ro["totarea"]), 1.0)
        if ro["status"] == 0:
            assert np.linalg.norm(cg - cg_o) <= 1e-6 * np.linalg.norm(cg_o)
    g.close()


@pytest.mark.parametrize("form", ["fp64", "fast"])
@pytest.mark.parametrize("nrows,lmax,points", [(2, 1, 127), (3, 2, 129), (5, 4, 130), (6, 6, 66)])
def test_jacobian_rows_at_any_scattering(native, oracle_lib, tmp_path, form, nrows, lmax, points):
    """Every row and column of J, with scattering coefficients that a fit does
    not take: the reference-order form's quotients must round like divisions
    there too.  Points around the 128 of a pass; coefficient counts with and
    without padding (4, 9, 25, 49 of 8, 16, 32, 56)."""
    w = synth.make_workload("jac", 60 + lmax, dense_lcs=1, dense_pts=20, sparse_pts=points - 20, years=6, true_lmax=2,
                            fit_lmax=lmax, nrows=nrows, noise=0.02, n_periods=2)
    path = synth.write_input(w, str(tmp_path))
    o = oracle_lib.Oracle(path)
    o.set_conw_r(o.conw_r)
    g = native.PeriodSearch(path, form={"fp64": native.PS_FORM_FP64, "fast": native.PS_FORM_FAST}[form])
    g.set_conw_r(o.conw_r)
    a = o.initial_parameters(o.freq(1), 6)
    C = g.ncoef
    for log_cl, cls in ((np.log(0.1), 1.0), (-3.0, 0.0), (0.7, 3.7e5), (-1.0, 1e-12)):
        a[C + 6], a[C + 7] = log_cl, cls
        y_o, J_o = o.model(a)
        y, J = g.model(a)
        assert np.linalg.norm(y - y_o) <= 1e-11 * np.linalg.norm(y_o)
        for k in range(g.ma):
            # a column may be what cancellation leaves: its scale is J's at least
            scale = max(np.linalg.norm(J_o[:, k]), 1e-3 * np.linalg.norm(J_o) / np.sqrt(g.ma))
            assert np.linalg.norm(J[:, k] - J_o[:, k]) <= 1e-11 * scale, (log_cl, cls, k)
    g.close()


def test_jacobian_of_an_overflowing_shape(native, oracle_lib):
    """Facet areas of 1e204: the reference-order form's sums then take the
    branch that leaves facets out which a point does not see."""
    path = golden_path("tiny")
    o = oracle_lib.Oracle(path)
    o.set_conw_r(o.conw_r)
    g = native.PeriodSearch(path, form=native.PS_FORM_FP64)
    g.set_conw_r(o.conw_r)
    a = o.initial_parameters(o.freq(1), 2)
    a[0] = 470.0
    y_o, J_o = o.model(a)
    y, J = g.model(a)
    # the products of the relative-lightcurve normalisation overflow: the same
    # entries must, and the others agree
    fine = np.isfinite(J_o)
    assert np.array_equal(fine, np.isfinite(J)) and np.abs(J_o[fine]).max() > 1e200 and np.all(np.isfinite(y_o))
    top = np.abs(J_o[fine]).max()
    for got, ref, ok in [(y, y_o, np.isfinite(y_o))] + [(J[:, k], J_o[:, k], fine[:, k]) for k in range(g.ma)]:
        # an exponent of 470 carries 470 roundings of exp's argument: 1e-13; a
        # column may be what cancellation leaves
        if ok.any():
            assert np.abs(got[ok] - ref[ok]).max() <= 1e-9 * max(np.abs(ref[ok]).max(), 1e-6 * top)
    g.close()
