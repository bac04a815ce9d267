"""The model pass takes four facets at a time, without branches, and (in the
reference-order form) divides through one reciprocal per pair: the trial points
of a fit must still follow the oracle's path.  Sizes at the edges: 8 nrows^2
facets around the staged chunk of 128 and its blocks of four, point counts
around a warp, a block of 256 threads and the four points a thread takes."""
import numpy as np
import pytest

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
