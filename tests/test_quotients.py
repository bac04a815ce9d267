"""The fit kernels' branch-free reciprocal and quotients (ps_fit_common.cuh)
against CUDA's division, bit for bit: the reference-order form's results rest on
their rounding.  Divisors over (2e-8, 4], numerators as mu, mu0 and the
Lommel-Seeliger coefficient take them, mantissas near all ones and all zeros,
and the operands whose quotients come closest to the middle of two numbers
(A 2^s = D (2 M + 1) +- k for small k)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

SRC = os.path.join(REPO, "tests", "quotient_selftest.cu")
HDR = os.path.join(REPO, "periodsearch_b200", "csrc", "ps_fit_common.cuh")
LIB = os.path.join(REPO, "tests", "_build", "libquotient_selftest.so")


def _lib():
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(SRC), os.path.getmtime(HDR)):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run(["nvcc", "-shared", "-std=c++17", "-Xcompiler", "-fPIC", "-O3", "-fmad=false", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-o", LIB, SRC], check=True)
    return ctypes.CDLL(LIB)


def _quotients(a, d):
    a, d = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(d, np.float64)
    out = np.empty((5, a.size))
    p = lambda x: x.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    assert _lib().quotient_selftest(p(a), p(d), a.size, p(out)) == 0
    return out


def _middles(rng, n):
    """(a, d) with quotients a hair from the middle of two numbers."""
    a, d = [], []
    while len(a) < n:
        D = int(rng.integers(1 << 52, 1 << 53)) | 1
        if len(a) % 4 == 0:  # mantissas near all ones
            D = (1 << 53) - int(rng.integers(1, 1 << 20)) | 1
        k = int(rng.integers(-8, 8)) * 2 + 1
        s = 53 + int(rng.integers(0, 2))
        M = -k * pow(D, -1, 1 << s) % (1 << s)  # odd: D M = -k mod 2^s
        M += (1 << 53) if M < 1 << 53 else 0
        if M >= 1 << 54 or (D * M + k) % (1 << s):
            continue
        A = (D * M + k) >> s
        if 1 << 52 <= A < 1 << 53:
            a.append(A * 2.0**-53)
            d.append(D * 2.0**-53)
    return np.array(a), np.array(d)


def _divisors(rng, n):
    d = np.exp(rng.uniform(np.log(2e-8), np.log(4.0), n))
    k = np.arange(n // 4)
    near = np.ldexp(2.0 - np.ldexp(1.0 + k % 4096, -52), rng.integers(-26, 1, k.size))  # just below a power of two
    over = np.ldexp(1.0 + np.ldexp(1.0 * (k % 4096), -52), rng.integers(-25, 2, k.size))  # at and just above one
    return np.concatenate([d, near, over])


def test_random_operands():
    rng = np.random.default_rng(1)
    d = _divisors(rng, 1 << 20)
    near_one = rng.choice([1.0, 2.0, 0.5, 1 + 2.0**-52, 1 - 2.0**-53, 2 - 2.0**-52], d.size)
    for a in (d * rng.uniform(0, 1, d.size), rng.uniform(1e-8, 2, d.size), near_one, -near_one, np.zeros(d.size),
              np.exp(rng.uniform(-460, 460, d.size)) * rng.choice([-1.0, 1.0], d.size)):
        q, q_ref, y, y_ref, y_newton = _quotients(a, d)
        assert np.array_equal(q, q_ref)
        assert np.array_equal(y, y_ref)
        assert np.max(np.abs(y_newton - y_ref) / np.spacing(y_ref)) <= 1


def test_numerators_out_of_the_ordinary():
    """Beyond 1e200 in size or below 1e-200, infinite, not a number: the division's
    quotient, a subnormal one to its spacing."""
    rng = np.random.default_rng(3)
    d = _divisors(rng, 1 << 16)
    tiny, huge = 10.0 ** rng.uniform(-323, -200, d.size), 10.0 ** rng.uniform(200, 308, d.size)
    for a in (tiny, -tiny, huge, -huge):
        q, q_ref, *_ = _quotients(a, d)
        sub = np.abs(q_ref) < 2.3e-308
        assert np.array_equal(q[~sub], q_ref[~sub])
        assert np.abs(q[sub] - q_ref[sub]).max(initial=0.0) <= 5e-324
    for a in (np.inf, -np.inf, np.nan):
        q, q_ref, *_ = _quotients(np.full(d.size, a), d)
        assert np.array_equal(q, q_ref, equal_nan=True)


def test_quotients_near_a_middle():
    rng = np.random.default_rng(2)
    a, d = _middles(rng, 200_000)
    for e in (0, -13, 2):
        q, q_ref, y, y_ref, _ = _quotients(a, d * 2.0**e)
        assert np.array_equal(q, q_ref)
        assert np.array_equal(y, y_ref)
