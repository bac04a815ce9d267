"""Matrix-free kernels at the edges of their splits: facet grids of one orbit
to several slices of antipodal pairs, point counts around a block of 32, 128
and 256, relative and calibrated lightcurves, parameters at which facets lie at
grazing incidence.  Bars as for the larger shapes: chi2, beta and products
agree with the explicit evaluation to 1e-10; a batch of unit vectors (the
Jacobian-free fit) with the oracle's fit to 1e-9."""
import numpy as np
import pytest

from conftest import golden_path
from periodsearch_b200 import synth

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("nrows,lmax,dense,points", [(1, 1, 0, 31), (2, 2, 1, 129), (4, 3, 2, 257), (6, 5, 0, 600),
                                                     (9, 6, 5, 1024)])
def test_products_and_gradient(native, oracle_lib, tmp_path, nrows, lmax, dense, points):
    w = synth.make_workload("adj", 80 + nrows, dense_lcs=dense, dense_pts=40, sparse_pts=points - 40 * dense, years=6,
                            true_lmax=2, fit_lmax=lmax, nrows=nrows, noise=0.02, n_periods=2)
    path = synth.write_input(w, str(tmp_path))
    o = oracle_lib.Oracle(path)
    o.set_conw_r(o.conw_r)
    g = native.PeriodSearch(path, form=native.PS_FORM_FAST)
    g.set_conw_r(o.conw_r)
    rng = np.random.default_rng(nrows)
    for pole in (1, 7):
        a = o.initial_parameters(o.freq(1), pole)
        alpha, beta, x2 = o.mrqcof(a)
        x2_g, beta_g = g.chi2_grad(a)
        assert abs(x2_g - x2) <= TOL * abs(x2)
        assert np.linalg.norm(beta_g - beta) <= TOL * np.linalg.norm(beta)
        v = rng.normal(size=g.mfit) / np.sqrt(np.maximum(np.diag(alpha), 1e-300))
        ref = alpha @ v
        # the product's scale: what its terms add up from
        scale = np.linalg.norm(np.abs(alpha) @ np.abs(v))
        assert np.linalg.norm(g.gn_product(a, v) - ref) <= TOL * scale
    g.close()


def test_calls_in_turn_do_not_leak(native, oracle_lib):
    """Gradient, product and Jacobian-free fit share one work buffer of
    different layouts: each result is the same after any of the others."""
    path = golden_path("tiny")
    o = oracle_lib.Oracle(path)
    o.set_conw_r(o.conw_r)
    g = native.PeriodSearch(path, form=native.PS_FORM_FP64)
    g.set_conw_r(o.conw_r)
    a = o.initial_parameters(o.freq(1), 3)
    v = np.ones(g.mfit)
    grad, prod = g.chi2_grad(a), g.gn_product(a, v)
    fit = g.fit_jfree(o.freq(2), 4)
    again = g.chi2_grad(a)
    assert again[0] == grad[0] and np.array_equal(again[1], grad[1])
    assert np.array_equal(g.gn_product(a, v), prod)
    assert g.fit_jfree(o.freq(2), 4) == fit
    g.close()
