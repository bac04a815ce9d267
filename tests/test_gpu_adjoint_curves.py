"""Matrix-free calls on relative lightcurves of every kind, against the explicit
evaluation of the reference-order form (ps_mrqcof) on the same arrays: sigmas
that differ within a curve, curves longer than the blocks the kernels take rows
in.  Bars as for the other shapes: 1e-10 of what the sums add up from."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _desc(seed, curves, lmax, nrows, vary_sigma):
    """Arrays of a problem with `curves` (relative, points) and directions within
    30 degrees of one another."""
    g = np.random.default_rng(seed)
    n = sum(k for _, k in curves)
    unit = lambda x: x / np.linalg.norm(x, axis=1, keepdims=True)  # noqa: E731
    ee = unit(g.normal(size=(n, 3)))
    ee0 = unit(ee + 0.25 * g.normal(size=(n, 3)) / np.sqrt(3))
    bright = g.uniform(0.5, 1.5, n)
    sig, at = np.empty(n), 0
    for _, k in curves:
        sig[at:at + k] = bright[at:at + k].mean() * (g.uniform(0.5, 2.0, k) if vary_sigma else 1.0)
        at += k
    tim = np.sort(g.uniform(0, 3000, n))
    return dict(lc_points=[k for _, k in curves], lc_relative=[r for r, _ in curves], tim=tim, ee=ee, ee0=ee0,
                brightness=bright, sig=sig, weight=g.uniform(0.5, 1.5, n), per_start=8.001, per_step_coef=0.5,
                per_end=7.999, ia_prd=1, phi0_rad=0.0, conw=0.1, lmax=lmax, mmax=lmax, nrows=nrows, par=[0.5, 0.1, -0.5],
                ia_par=[1, 1, 1], cl=0.1, ia_cl=1, stop_condition=5.0, n_iter_min=5, alamda_incr=5.0, alamda_start=0.1,
                jd_min=float(tim[0]), jd_max=float(tim[-1]), escl=0.6)


def _check(native, desc, seed):
    g = native.PeriodSearch(desc=desc, form=native.PS_FORM_FAST)
    e = native.PeriodSearch(desc=desc, form=native.PS_FORM_FP64)
    for c in (g, e):
        c.set_conw_r(0.4)
    rng = np.random.default_rng(seed)
    C = g.ncoef
    for pole in (0.4, 2.1):
        a = np.concatenate([g.array("cg_first"), [pole, 1.0, 24 * 2 * np.pi * g.freq_start, 0.5, 0.1, -0.5, np.log(0.1), 1.0]])
        a[:C] += 0.02 * rng.normal(size=C) / np.maximum(np.abs(g.array("dsph").reshape(-1, C)).max(axis=0), 1)
        alpha, beta, x2 = e.mrqcof(a)
        x2_g, beta_g = g.chi2_grad(a)
        assert abs(x2_g - x2) <= TOL * abs(x2)
        # beta sums weighted residuals, of size sqrt(chi2), times J's columns, of
        # size sqrt(alpha_kk)
        scale = np.sqrt(np.diag(alpha) * x2)
        assert np.all(np.abs(beta_g - beta) <= TOL * scale)
        v = rng.normal(size=g.mfit) / np.sqrt(np.maximum(np.diag(alpha), 1e-300))
        got, ref = g.gn_product(a, v), alpha @ v
        assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(np.abs(alpha) @ np.abs(v))
    g.close()
    e.close()


@pytest.mark.parametrize("curves,lmax,nrows", [([(1, 40)], 2, 3), ([(1, 63), (0, 70), (1, 65)], 3, 4),
                                               ([(0, 30), (1, 1), (1, 300)], 4, 5)])
def test_sigma_varying_within_a_curve(native, curves, lmax, nrows):
    _check(native, _desc(3, curves, lmax, nrows, True), 4)


@pytest.mark.parametrize("curves,lmax,nrows", [([(1, 64)], 2, 3), ([(1, 65), (0, 70), (1, 128)], 3, 4), ([(0, 64), (1, 129)], 3, 4),
                                               ([(1, 255), (1, 256), (0, 257), (1, 700)], 4, 5), ([(1, 5000)], 6, 10)])
def test_curves_longer_than_a_block(native, curves, lmax, nrows):
    _check(native, _desc(5, curves, lmax, nrows, False), 6)


def test_time_of_a_long_relative_curve(native):
    """The rows of one long relative lightcurve spread over the GPU like those of
    calibrated points: a gradient costs 1.6 times as much on it (nine times when one
    CTA formed them in turn)."""
    us = {}
    for rel in (0, 1):
        g = native.PeriodSearch(desc=_desc(7, [(rel, 20000)], 6, 10, False), form=native.PS_FORM_FAST)
        g.set_conw_r(0.4)
        a = np.concatenate([g.array("cg_first"), [0.4, 1.0, 24 * 2 * np.pi * g.freq_start, 0.5, 0.1, -0.5, np.log(0.1), 1.0]])
        g.chi2_grad(a)
        t = []
        for _ in range(9):
            t0 = time.perf_counter()
            g.chi2_grad(a)
            t.append(time.perf_counter() - t0)
        us[rel] = 1e6 * sorted(t)[2]
        g.close()
    print(f"gradient, 20 000 points, 800 facets: {us[0]:.0f} us calibrated, {us[1]:.0f} us on one relative curve")
    assert us[1] < 3 * us[0]


def test_work_memory_of_a_gradient(native):
    """A gradient takes work memory for one direction (16.5 MB at 20 000 points
    and 2048 facets), not for the batch of eight of a Jacobian-free fit (38 MB)."""
    torch = pytest.importorskip("torch")
    taken = []
    for points, nrows in ((60, 3), (20000, 16)):  # the first loads the kernels
        g = native.PeriodSearch(desc=_desc(8, [(0, points)], 3, nrows, False), form=native.PS_FORM_FAST)
        g.set_conw_r(0.4)
        a = np.concatenate([g.array("cg_first"), [0.4, 1.0, 24 * 2 * np.pi * g.freq_start, 0.5, 0.1, -0.5, np.log(0.1), 1.0]])
        native.load_library().ps_release_cached_memory()
        free = torch.cuda.mem_get_info()[0]
        g.chi2_grad(a)
        taken.append(free - torch.cuda.mem_get_info()[0])
        g.close()
    assert taken[1] < 24 << 20, taken
