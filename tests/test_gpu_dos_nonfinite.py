"""NaN energies in the Gaussian sums (csrc/gauss_sum.cuh) on a GB300.

A k-point whose overlap is not positive definite has NaN eigenvalues.  A sum without a window contains their terms, so
the whole curve is NaN; a window keeps the bands that compare as inside, so they drop out.  The grids take the power
recurrence, one exponential per point (coarse), and ragged ends.
"""
import types

import numpy as np
import pytest
import torch

from slakonet_gb300 import Geometry, compute_atom_projected_dos
from test_gpu_dos_fermi import _Batch, _dev, _dos

pytestmark = pytest.mark.gpu
SIZES = [(3, 4), (70, 5), (1, 40)]


def _with_nan(seed, bands):
    B = _Batch(SIZES, seed=seed)
    for e in B.eig[:2]:
        e[1, bands] = np.nan
    B.E = _dev(np.concatenate([e.reshape(-1) for e in B.eig]), torch.float64)
    return B


@pytest.mark.parametrize("npts", [1, 7, 300, 2000])
@pytest.mark.parametrize("bands", [slice(None), slice(2, 3)])
def test_a_nan_band_makes_the_whole_dos_nan_without_a_window(npts, bands):
    _, dos, _ = _dos(_with_nan(2, bands), [0.0] * 3, -20.0, 10.0, npts, 0.1, 0.0)
    assert np.isnan(dos[:2]).all() and np.isfinite(dos[2]).all()


@pytest.mark.parametrize("npts", [7, 300, 2000])
@pytest.mark.parametrize("window", [9.0, 40.0])
def test_a_failed_k_point_is_outside_every_window(npts, window):
    B = _with_nan(2, slice(None))
    _, dos, _ = _dos(B, [0.0] * 3, -20.0, 10.0, npts, 0.1, window)
    for s in range(2):                                  # at weight zero beside the same bands, finite
        B.eig[s][1] = B.eig[s][0]
        B.w[s][1] = 0.0
    B.E = _dev(np.concatenate([e.reshape(-1) for e in B.eig]), torch.float64)
    B.kw = _dev(np.concatenate(B.w), torch.float64)
    _, ref, _ = _dos(B, [0.0] * 3, -20.0, 10.0, npts, 0.1, window)
    assert np.array_equal(dos, ref)


def _pdos(eig, vec, fermi, npts, nk, nb):
    props = {"fermi_energy_eV": fermi,
             "calc": types.SimpleNamespace(eigenvalue=torch.as_tensor(eig)[None],
                                           eigenvectors=torch.as_tensor(vec).permute(1, 2, 0)[None])}
    geom = Geometry(np.array([14, 6]), np.zeros((2, 3)), np.eye(3) * 9.0)
    return compute_atom_projected_dos(props, geom, 0.1, (-8.0, 6.0), n_points=npts)[1]


@pytest.mark.parametrize("npts", [9, 1000])
def test_nan_energies_levels_and_vectors_make_the_projected_dos_nan(npts):
    rng = np.random.default_rng(3)
    nk, nb = 70, 8
    eig = np.sort(rng.uniform(-0.8, 0.7, (nk, nb)), axis=1)
    vec = rng.standard_normal((nk, nb, nb)) + 1j * rng.standard_normal((nk, nb, nb))
    assert all(np.isfinite(p).all() for p in _pdos(eig, vec, 0.0, npts, nk, nb).values())
    bad = eig.copy()
    bad[5] = np.nan                                     # a failed k-point; the Fermi level falls back to zero
    for args in ((bad, vec, 0.0), (eig, vec, float("nan"))):
        for p in _pdos(*args, npts, nk, nb).values():
            assert np.isnan(p).all()
    nanvec = vec.copy()
    nanvec[5] = np.nan
    for p in _pdos(eig, nanvec, 0.0, npts, nk, nb).values():
        assert np.isnan(p).all()
