"""The special functions behind the confidence bounds (csrc/nz_math.cuh),
compiled for the host: the finite sum that takes the place of the continued
fraction on one side, and the quantiles at the run counts where iterations
used to run on."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
D = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope='module')
def fns(tmp_path_factory):
    if shutil.which('g++') is None:
        pytest.skip('no host C++ compiler')
    d = tmp_path_factory.mktemp('q')
    (d / 'q.cpp').write_text(
        '#include <cmath>\n#define __host__\n#define __device__\nusing std::isfinite;\n#include "%s"\n'
        'extern "C" {\n'
        'void tails(const double *a, const double *b, const double *x, double *s, int n)'
        ' { for (int i = 0; i < n; ++i) s[i] = nz::binomial_sum(a[i], b[i], x[i], 1.0 - x[i], 1.0); }\n'
        'void bq(const double *q, const double *a, const double *b, double *o, int n)'
        ' { for (int i = 0; i < n; ++i) o[i] = nz::beta_quantile(q[i], a[i], b[i]); }\n'
        'void tq(const double *q, const double *v, double *o, int n)'
        ' { for (int i = 0; i < n; ++i) o[i] = nz::student_t_quantile(q[i], v[i]); }\n}\n'
        % os.path.join(REPO, 'pypercolate_gb300', 'csrc', 'nz_math.cuh'))
    so = str(d / 'q.so')
    subprocess.run(['g++', '-O2', '-std=c++17', '-shared', '-fPIC', str(d / 'q.cpp'), '-o', so], check=True)
    lib = ctypes.CDLL(so)

    def call(name, *arrays):
        arrays = [np.ascontiguousarray(v, dtype=np.float64) for v in arrays]
        getattr(lib, name)(*[v.ctypes.data_as(D) for v in arrays], ctypes.c_int(arrays[0].size))
        return arrays
    return call


@pytest.mark.parametrize('a', [1, 2, 3, 10, 100, 511, 4095, 4096])
@pytest.mark.parametrize('ratio', [8, 9, 100, 5000])
def test_binomial_sum_is_the_exact_tail(fns, a, ratio):
    """Without the common prefactor x^a y^b / B(a, b), from the mean to 10
    standard deviations above it, against all a terms in 40 digits: at most 596
    terms of 3 roundings of 2^-53 each, < 2e-13."""
    mp = pytest.importorskip('mpmath')
    b = float(a * ratio)
    mean = (a + 1.0) / (a + b + 2.0)
    sd = np.sqrt(a * b / ((a + b) ** 2 * (a + b + 1.0)))
    x = np.minimum(mean + sd * np.array([0.001, 0.5, 2.0, 10.0]), 0.9)
    s = fns('tails', np.full(x.size, a), np.full(x.size, b), x, np.empty(x.size))[-1]
    with mp.workdps(40):
        for got, xi in zip(s, x):
            odds, total, term = mp.mpf(1.0 - xi) / mp.mpf(xi), mp.mpf(0), mp.mpf(1)
            for m in range(a):
                total += term
                term *= mp.mpf(a - 1 - m) * odds / (b + 1 + m)
            assert abs(got / (total / (mp.mpf(b) * xi)) - 1) < 2e-13


@pytest.mark.parametrize('runs', [3, 40, 4000, 5000, 40000, 400000])
def test_beta_quantiles(fns, runs):
    st = pytest.importorskip('scipy.stats')
    rng = np.random.default_rng(runs)
    k = np.unique(np.concatenate([np.arange(0, min(runs, 12) + 1), runs - np.arange(0, min(runs, 12) + 1),
                                  rng.integers(0, runs + 1, 300)]))
    q, k = (v.ravel() for v in np.meshgrid([0.025, 0.975, 0.5, 1e-6], k))
    out = fns('bq', q, k + 1.0, runs - k + 1.0, np.empty(q.size))[-1]
    # lgamma near 1e6 keeps 1e-10 of the prefactor, in scipy as here
    np.testing.assert_allclose(out, st.beta.ppf(q, k + 1.0, runs - k + 1.0), rtol=1e-9)


def test_t_quantiles(fns):
    st = pytest.importorskip('scipy.stats')
    v = np.concatenate([np.arange(1.0, 40.0), [99, 999, 3999, 9998, 9999, 10000, 99999]])
    q, v = (w.ravel() for w in np.meshgrid([0.025, 0.975, 0.15865, 0.51, 1e-7], v))
    out = fns('tq', q, v, np.empty(q.size))[-1]
    np.testing.assert_allclose(out, st.t.ppf(q, v), rtol=1e-8)


@pytest.mark.parametrize('tail', [0.4, 0.15865, 0.025, 0.0005])
@pytest.mark.parametrize('v', [400, 700, 2000, 9999])
def test_t_expansion_where_it_applies(fns, tail, v):
    """Five terms leave < 1e-15; some ten roundings of 2^-53 and the normal
    quantile's own on top: < 1e-14.  (Tails of 0.0005 at v = 400 and 700 are
    iterated, with lgamma's 1e-13 of the prefactor.)"""
    mp = pytest.importorskip('mpmath')
    got = fns('tq', [1.0 - tail], [v], np.empty(1))[-1][0]
    with mp.workdps(30):
        tail = mp.mpf(1.0) - mp.mpf(1.0 - tail)
        z = mp.sqrt(2) * mp.erfinv(1 - 2 * tail)
        want = mp.findroot(lambda t: mp.betainc(mp.mpf(v) / 2, mp.mpf(1) / 2, 0, v / (v + t * t),
                                                regularized=True) / 2 - tail, z * (1 + (z * z + 1) / (4 * v)))
        assert abs(got / want - 1) < (1e-14 if tail > 0.001 or v >= 2000 else 1e-12)
