"""Width of the tridiagonal eigenvalue search's last bracket (csrc/sturm.cuh), built for the host.  Close eigenvalues are
bisected to 2e-15 of the norm and the middle is taken, 1e-15 off at most; a single one's last secant step is below 2e-15.
The count's rounding and LAPACK's are a few eps of the norm each (8 eps together here).  Symmetric spectra about zero and
eigenvalues that coincide are where the earlier width of 1e-14 showed."""
import numpy as np
import pytest
import scipy.linalg as sla

from test_sturm_host import search  # noqa: F401  (the fixture)

EPS = 2.2e-16


def _matrix(kind, rng):
    if kind == "pairs":                                       # two copies, coupled by nothing: each eigenvalue twice
        n = int(rng.integers(2, 40))
        d, e = rng.standard_normal(n), rng.standard_normal(n - 1)
        return np.r_[d, d], np.r_[e, 0.0, e]
    if kind == "nearly":                                      # a level with couplings far below the bracket
        n = int(rng.integers(3, 60))
        return np.full(n, rng.uniform(-1, 1)) + 1e-9 * rng.standard_normal(n), np.r_[1e-8 * rng.standard_normal(n - 2), 0.7]
    n = int(rng.integers(2, 120))
    return rng.standard_normal(n), rng.standard_normal(n - 1)


@pytest.mark.parametrize("kind", ["pairs", "nearly", "plain"])
def test_error_is_a_few_eps_of_the_norm(search, kind):        # noqa: F811
    for seed in range(20):
        d, e = _matrix(kind, np.random.default_rng(seed))
        got = search(d, e * e)
        ref = sla.eigvalsh_tridiagonal(d, np.abs(e)) if kind != "pairs" else \
            np.sort(np.repeat(sla.eigvalsh_tridiagonal(d[:len(d) // 2], np.abs(e[:len(d) // 2 - 1])), 2)) if len(d) > 2 \
            else np.sort(d)
        a = np.abs(e)
        norm = (np.abs(d) + np.r_[0, a] + np.r_[a, 0]).max()
        err = np.abs(got - ref).max()
        assert err <= (2e-15 + 8 * EPS) * norm, (kind, seed, err / norm)
