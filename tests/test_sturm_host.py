"""The tridiagonal eigenvalue search (csrc/sturm.cuh), built for the host, against LAPACK on matrices where a search goes
wrong: graded ones (an eigenvalue just outside a bracket once passed for the one inside), clusters, zero couplings,
exact integers, large and small scales.  Error relative to the norm: the last bracket's width, 1e-14, and the count's
own rounding, a few eps per row entering as perturbations of the entries: 1e-14 + 10 eps."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.linalg as sla

from conftest import ROOT

SHIM = """#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
using std::max;
using std::min;
#define __device__
#define __forceinline__ inline
static inline long long __double_as_longlong(double v) { long long r; std::memcpy(&r, &v, 8); return r; }
static inline double __longlong_as_double(long long v) { double r; std::memcpy(&r, &v, 8); return r; }
static inline int __double2hiint(double v) { return (int)(__double_as_longlong(v) >> 32); }
static inline int __double2loint(double v) { return (int)__double_as_longlong(v); }
static inline double __hiloint2double(int h, int l) { return __longlong_as_double(((long long)h << 32) | (unsigned)l); }
static inline bool is_zero_bits(double v) { return ((unsigned long long)__double_as_longlong(v) << 1) == 0; }
static inline double flip_sign(double v) { return -v; }
"""


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("sturm")
    shutil.copy(os.path.join(ROOT, "slakonet_gb300", "csrc", "sturm.cuh"), d)
    shutil.copy(os.path.join(ROOT, "tests", "sturm_check.cpp"), d)
    (d / "skn_common.cuh").write_text(SHIM)
    exe = str(d / "sturm_check")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-w", str(d / "sturm_check.cpp"), "-o", exe])

    def run(d_, e2):
        text = "\n".join([str(len(d_)), " ".join("%.17g" % x for x in d_), " ".join("%.17g" % x for x in e2), ""])
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        return np.array([float(x) for x in out.split()])
    return run


def _matrix(kind, rng):
    n = int(rng.integers(2, 140))
    if kind == "graded":
        X = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        D = np.logspace(0, -rng.uniform(1, 9), n)
        T = sla.hessenberg(D[:, None] * (X + X.conj().T) / 2 * D[None])
        return np.real(np.diag(T)).copy(), np.abs(np.diag(T, -1)) ** 2
    if kind == "scattered":
        return rng.standard_normal(n) * 10.0 ** rng.uniform(-8, 0, n), 10.0 ** rng.uniform(-18, 0, n - 1)
    if kind == "wilkinson":
        return np.abs(np.arange(n) - (n - 1) / 2), np.ones(n - 1)
    if kind == "integers":
        return rng.integers(-3, 4, n).astype(float), rng.integers(0, 2, n - 1).astype(float)
    s = 2.0 ** float(rng.integers(-300, 300))
    return s * rng.standard_normal(n), s * s * rng.chisquare(4, n - 1)


@pytest.mark.parametrize("kind", ["graded", "scattered", "wilkinson", "integers", "scaled"])
def test_eigenvalues_agree_with_lapack(search, kind):
    for seed in range(12):
        d, e2 = _matrix(kind, np.random.default_rng(seed))
        ref = np.sort(sla.eigvalsh_tridiagonal(d, np.sqrt(e2)))
        err = np.abs(search(d, e2) - ref).max()
        norm = (np.abs(d) + np.sqrt(np.r_[0, e2]) + np.sqrt(np.r_[e2, 0])).max()       # what the search's widths refer to
        assert err <= (1e-14 + 10 * 2.2e-16) * norm, (kind, seed, err / norm)


def test_the_graded_matrix_that_went_wrong(search):
    rng = np.random.default_rng(1)
    n = 100
    X = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    Y = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * 0.3
    D = np.logspace(0, -6, n)
    H, S = D[:, None] * (X + X.conj().T) / 2 * D[None], np.eye(n) + Y @ Y.conj().T / n
    L = np.linalg.cholesky(S)
    C = sla.solve_triangular(L, sla.solve_triangular(L, H, lower=True).conj().T, lower=True).conj().T
    T = sla.hessenberg((C + C.conj().T) / 2)
    d, e2 = np.real(np.diag(T)).copy(), np.abs(np.diag(T, -1)) ** 2
    ref = np.sort(sla.eigvalsh_tridiagonal(d, np.sqrt(e2)))
    assert np.abs(search(d, e2) - ref).max() <= 1.3e-14 * np.abs(ref).max() * 3.0
