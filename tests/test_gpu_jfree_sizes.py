"""Jacobian-free fits at the edges of the kernels' splits: free parameters below,
at and above multiples of the eight directions of a batch, facet grids of one
orbit to several slices, lightcurves shorter and longer than a block of 64 points.
Fits of eight steps, whose rounding differences stay near 1e-12, to the bars of the
other fits against the oracle."""
import numpy as np
import pytest

from periodsearch_b200 import synth

pytestmark = pytest.mark.gpu

FIT_TOL = 1e-9


@pytest.mark.parametrize("nrows,lmax,dense,per,points,free_cl,mfit",
                         [(1, 1, 0, 0, 31, 0, 10), (3, 2, 1, 64, 130, 1, 16), (4, 3, 2, 40, 257, 0, 22),
                          (6, 4, 1, 65, 300, 1, 32), (7, 5, 1, 300, 420, 1, 43), (9, 6, 2, 129, 1024, 0, 55)])
def test_fits_match_the_oracle(native, oracle_lib, tmp_path, nrows, lmax, dense, per, points, free_cl, mfit):
    w = synth.make_workload("jf", 50 + nrows, dense_lcs=dense, dense_pts=per, sparse_pts=points - dense * per, years=6,
                            true_lmax=2, fit_lmax=lmax, nrows=nrows, noise=0.02, n_periods=2, stop_condition=8)
    path = synth.write_input(w, str(tmp_path))
    lines = open(path).read().splitlines(True)
    value = lines[9].split()[0]
    lines[9] = "%s %d\n" % (value, free_cl)
    open(path, "w").write("".join(lines))
    o = oracle_lib.Oracle(path)
    o.set_conw_r(o.conw_r)
    g = native.PeriodSearch(path, form=native.PS_FORM_FAST)
    g.set_conw_r(o.conw_r)
    assert g.mfit == mfit
    for pole in (1, 6):
        ro, cg_o = o.fit(o.freq(1), pole)
        rj, cg = g.fit_jfree(o.freq(1), pole, params=True)
        assert rj["niter"] == int(ro["niter"]) and rj["status"] == int(ro["status"])
        assert abs(rj["chisq"] - ro["chisq"]) <= FIT_TOL * abs(ro["chisq"])
        assert abs(rj["totarea"] - ro["totarea"]) <= FIT_TOL * abs(ro["totarea"])
        assert abs(rj["lambda_deg"] - ro["lambda_deg"]) <= 1e-6 and abs(rj["beta_deg"] - ro["beta_deg"]) <= 1e-6
        if ro["status"] == 0:
            assert np.linalg.norm(cg - cg_o) <= 1e-6 * np.linalg.norm(cg_o)
    g.close()
