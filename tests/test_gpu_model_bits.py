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
