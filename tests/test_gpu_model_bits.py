"""In the reference-order form the model pass of a trial point forms chi2 with the
operations and sum orders of the full evaluation: a fit's chi2 (its last accepted
point's, from the model pass) has the bits that one evaluation at the fit's
parameters gives.  (The fast form's evaluation sums a point's facets in four
parts, its model pass in one.)"""
import numpy as np
import pytest

from periodsearch_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrows,lmax,dense,points", [(1, 1, 0, 33), (4, 2, 1, 257), (6, 3, 2, 300), (10, 6, 2, 760),
                                                     (9, 7, 1, 500)])
def test_fit_chi2_equals_the_evaluation_bit_for_bit(native, tmp_path, nrows, lmax, dense, points):
    w = synth.make_workload("bits", 20 + nrows, dense_lcs=dense, dense_pts=50, sparse_pts=points - 50 * dense, years=6,
                            true_lmax=2, fit_lmax=lmax, nrows=nrows, noise=0.02, n_periods=3, stop_condition=9)
    path = synth.write_input(w, str(tmp_path))
    g = native.PeriodSearch(path, form=native.PS_FORM_FP64)
    g.set_conw_r(g.conw_r)
    for pole in range(1, 11):
        r, cg = g.fit(g.freq_start, pole, params=True)
        assert np.isfinite(r["chisq"])
        assert g.mrqcof(cg)[2] == r["chisq"], pole
    g.close()


def test_scattering_coefficients_out_of_the_ordinary(native, oracle_lib, tmp_path):
    """Rows at Lommel-Seeliger coefficients whose quotients overflow, vanish or are
    not numbers are what the oracle's divisions give.  (The data points' rows: the
    convexity rows do not depend on the coefficient.)"""
    w = synth.make_workload("odd", 31, dense_lcs=0, dense_pts=0, sparse_pts=140, years=6, true_lmax=2, fit_lmax=2,
                            nrows=4, noise=0.02, n_periods=2)
    path = synth.write_input(w, str(tmp_path))
    o = oracle_lib.Oracle(path)
    o.set_conw_r(o.conw_r)
    g = native.PeriodSearch(path, form=native.PS_FORM_FP64)
    g.set_conw_r(o.conw_r)
    a = o.initial_parameters(o.freq(1), 3)
    C = g.ncoef
    for log_cl, cls in ((-2.0, 1e305), (-2.0, 1.7e308), (-800.0, 1e-305), (-800.0, 4e-308), (-800.0, 5e-324),
                        (-2.0, 0.0), (-2.0, np.inf), (-2.0, -np.inf), (-2.0, np.nan)):
        a[C + 6], a[C + 7] = log_cl, cls
        y_o, J_o = o.model(a)
        y, J = g.model(a)
        for got, ref in ((y[:-3], y_o[:-3]), (J[:-3], J_o[:-3])):
            assert np.array_equal(np.isnan(got), np.isnan(ref)), (log_cl, cls)
            assert np.array_equal(np.isposinf(got), np.isposinf(ref)), (log_cl, cls)
            assert np.array_equal(np.isneginf(got), np.isneginf(ref)), (log_cl, cls)
            fine = np.isfinite(ref)
            # subnormal values have no more than their spacing
            err = np.abs(got[fine] - ref[fine])
            assert np.all(err <= 1e-11 * np.abs(ref[fine]).max(initial=0.0) + 1e3 * 5e-324), (log_cl, cls)
    g.close()
