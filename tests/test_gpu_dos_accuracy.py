"""Accuracy of the Gaussian sums (csrc/gauss_sum.cuh) on a GB300 against sums in extended precision at the grid's own points.

Relative error of one Gaussian at t = (x - e) / sigma on a lane's j-th point (j <= 7, d = step / sigma), eps = 2^-52: t is
rounded twice beside the rounding of E - mu, so t^2 / 2 and the exponential give (1.5 t^2 + 1) eps; the power's base is off
by (1 + |t| d) eps, j times, its products by j / 2 eps, the last factor by 3 eps.  E - mu is exact or off by
(eps / 2) |E - mu| H2E / sigma in t.  Nothing grows with |x|, or with the Fermi level's own size."""
import numpy as np
import pytest
import torch

from test_gpu_dos_fermi import H2E, _Batch, _dev, _dos

pytestmark = pytest.mark.gpu
LD = np.longdouble
EPS = 2.0 ** -52


def _reference(grid, e, mu, sigma):
    t = (grid.astype(LD) - (LD(e) - LD(mu)) * LD(H2E)) / LD(sigma)
    return np.exp(-t * t / 2) / (LD(sigma) * np.sqrt(2 * LD(np.pi))), np.abs(t.astype(float))


@pytest.mark.parametrize("lo,hi,npts,sigma", [(-8.0, 6.0, 1000, 0.05), (-10.0, 10.0, 5000, 0.1), (-20.0, 10.0, 1000, 0.1),
                                              (-20.0, 10.0, 40, 0.1)])
@pytest.mark.parametrize("mu", [0.0, -5.0])
def test_one_band_at_the_points_of_the_grid(lo, hi, npts, sigma, mu):
    n = 60
    B = _Batch([(1, 1)] * n, seed=npts)
    e = np.random.default_rng(4).uniform(0.9 * lo, 0.9 * hi, n) / H2E + mu
    B.E = _dev(e, torch.float64)
    grid, dos, _ = _dos(B, [mu] * n, lo, hi, npts, sigma, 0.0)
    d = (hi - lo) / (npts - 1) / sigma
    for s in range(n):
        ref, t = _reference(grid, e[s], mu, sigma)
        near = t <= 4.0
        shift = 0.5 * EPS * abs(e[s] - mu) * H2E / sigma
        bound = EPS * (1.5 * t * t + 1.0 + 7.0 * (1.0 + t * d) + 3.5 + 3.0 + 1.0) + t * shift
        err = np.abs((dos[s][near] - ref[near]) / ref[near]).astype(float)
        assert (err <= bound[near]).all(), (s, (err / bound[near]).max())
