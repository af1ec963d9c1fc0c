"""DOS and Fermi kernels at the sizes where their splits change (needs a GB300).

The DOS kernel gives 8 grid points to a lane, 64 to a tile, 256 to a CTA, and cuts the bands into 64 slices
(whole k-points from 64 k-points up, parts of a k-point below); fine grids take the power recurrence, coarse ones
one exponential per point.  The Fermi kernel deals blocks of 256 eigenvalues to up to 16 CTAs.
"""
import numpy as np
import pytest
import torch

from oracle import slako_oracle as O
from slakonet_gb300._lib import call, ptr

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
H2E = 27.211


def _dev(a, dtype):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=DEV)


class _Batch:
    def __init__(self, sizes, seed, lo=-0.8, hi=0.7):
        rng = np.random.default_rng(seed)
        self.eig = [np.sort(rng.uniform(lo, hi, (nk, nb)), axis=1) for nk, nb in sizes]
        self.w = [rng.uniform(0.5, 1.5, nk) for nk, _ in sizes]
        self.w = [x / x.sum() for x in self.w]
        self.ne = [float(max(1, nb)) for _, nb in sizes]          # half filling
        cnt = [e.size for e in self.eig]
        i64, i32, f64 = torch.int64, torch.int32, torch.float64
        self.off = _dev(np.concatenate([[0], np.cumsum(cnt)[:-1]]), i64)
        self.nk = _dev([s[0] for s in sizes], i32)
        self.nb = _dev([s[1] for s in sizes], i32)
        self.kwo = _dev(np.concatenate([[0], np.cumsum([s[0] for s in sizes])[:-1]]), i64)
        self.kw = _dev(np.concatenate(self.w), f64)
        self.E = _dev(np.concatenate([e.reshape(-1) for e in self.eig]), f64)
        self.nel = _dev(self.ne, f64)
        self.n = len(sizes)


def _dos(B, mu, lo, hi, npts, sigma, window):
    m = _dev(mu, torch.float64)
    grid = torch.empty(npts, dtype=torch.float64, device=DEV)
    dos = torch.empty(B.n, npts, dtype=torch.float64, device=DEV)
    stats = torch.zeros(B.n, 24, dtype=torch.float64, device=DEV)
    call("skn_dos", B.n, ptr(B.off), ptr(B.nk), ptr(B.nb), ptr(B.kwo), ptr(B.kw), ptr(B.E), ptr(m), lo, hi, npts,
         sigma, window, ptr(grid), ptr(dos), ptr(stats), torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize()
    return grid.cpu().numpy(), dos.cpu().numpy(), stats.cpu().numpy()


SIZES = [(1, 1), (1, 130), (2, 37), (5, 9), (31, 4), (63, 3), (64, 5), (65, 2), (200, 7)]


@pytest.mark.parametrize("npts", [1, 2, 7, 63, 64, 65, 256, 257, 1000, 5000])
@pytest.mark.parametrize("window,sigma", [(0.0, 0.1), (9.0, 0.1), (0.0, 0.05), (40.0, 0.05), (3.0, 0.3)])
def test_dos_matches_direct_sum(npts, window, sigma):
    """Relative error of a Gaussian: |t| dt with dt the rounding of the energies over sigma (40 eV 2^-53 * 4 / 0.05
    = 4e-13) and |t| <= 38.8, so 2e-11 of a sum of non-negative terms; a point within rounding of a window's edge
    may keep or drop a band, at most 4 exp(-window^2 / 2) / (sigma sqrt(2 pi)) in all."""
    B = _Batch(SIZES, seed=npts)
    mu = [0.01 * i for i in range(B.n)]
    grid, dos, stats = _dos(B, mu, -20.0, 10.0, npts, sigma, window)
    norm = 1.0 / (sigma * np.sqrt(2.0 * np.pi))
    atol = 1e-290 + (4.0 * norm * np.exp(-0.5 * window ** 2) if window > 0 else 0.0)
    for s in range(B.n):
        ev = (B.eig[s] - mu[s]) * H2E
        t = (grid[:, None, None] - ev[None]) / sigma
        g = np.exp(-0.5 * t * t) * norm
        if window > 0:
            g = np.where((ev[None] >= grid[:, None, None] - window * sigma) &
                         (ev[None] <= grid[:, None, None] + window * sigma), g, 0.0)
        ref = np.einsum("pkb,k->p", g, B.w[s])
        np.testing.assert_allclose(dos[s], ref, rtol=2e-11, atol=atol)
    if npts > 1:
        np.testing.assert_array_equal(grid, torch.linspace(-20.0, 10.0, npts, dtype=torch.float64).numpy())


def test_dos_of_a_structure_does_not_depend_on_the_batch():
    B = _Batch(SIZES, seed=3)
    mu = [0.01 * i for i in range(B.n)]
    for window in (0.0, 9.0):
        _, dos, _ = _dos(B, mu, -20.0, 10.0, 1000, 0.1, window)
        for s in (1, 4, 8):
            one = _Batch([SIZES[s]], seed=0)
            one.E, one.kw = _dev(B.eig[s].reshape(-1), torch.float64), _dev(B.w[s], torch.float64)
            _, alone, _ = _dos(one, [mu[s]], -20.0, 10.0, 1000, 0.1, window)
            assert np.array_equal(alone[0], dos[s])


def test_nan_fermi_level_gives_a_nan_dos():
    B = _Batch([(3, 4), (3, 4)], seed=1)
    _, dos, _ = _dos(B, [np.nan, 0.0], -20.0, 10.0, 300, 0.1, 9.0)
    assert np.isnan(dos[0]).all() and np.isfinite(dos[1]).all()


def test_fermi_and_gap_over_the_split_sizes():
    """Blocks of 256 eigenvalues: one below, at and above each edge, up to more than 16 blocks.  The spectra are
    dense (metals), where the search contracts, so its level agrees with the oracle's to its own stopping
    accuracy; the band edges are compared at the kernel's own level, where both sides do the same operations."""
    sizes = [(1, 1), (1, 8), (15, 17), (8, 32), (1, 257), (7, 73), (27, 19), (41, 25), (63, 65), (64, 64), (97, 85), (500, 40)]
    B = _Batch(sizes, seed=5)
    mu = torch.empty(B.n, dtype=torch.float64, device=DEV)
    stats = torch.zeros(B.n, 24, dtype=torch.float64, device=DEV)
    st = torch.empty(B.n, dtype=torch.int32, device=DEV)
    call("skn_fermi_gap", B.n, ptr(B.off), ptr(B.nk), ptr(B.nb), ptr(B.kwo), ptr(B.kw), ptr(B.nel), ptr(B.E), 0.01,
         1e-6, 100, ptr(mu), ptr(stats), ptr(st), torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize()
    stats, mu, st = stats.cpu().numpy(), mu.cpu().numpy(), st.cpu().numpy()
    for s in range(B.n):
        ref, it, conv = O.fermi_search(B.eig[s], B.w[s], B.ne[s])
        assert (st[s] == 0) == conv
        if np.isfinite(ref):
            assert abs(mu[s] - ref) <= 1e-9 * max(1.0, abs(ref)), (sizes[s], mu[s], ref)
        else:
            assert not np.isfinite(mu[s])
            continue
        bs = O.band_structure_props(B.eig[s], mu[s])
        be = O.band_energy(B.eig[s], B.w[s], mu[s])
        assert abs(stats[s][23] - be) <= 1e-12 * B.eig[s].size
        rel = (B.eig[s] - mu[s]) * H2E
        v, c = rel[rel < 0], rel[rel >= 0]
        assert stats[s][8] == (v.max() - v.min() if len(v) else 0.0)
        assert stats[s][9] == (c.max() - c.min() if len(c) else 0.0)
        kv = np.where(rel < 0, rel, -np.inf).max(1)
        kc = np.where(rel > 0, rel, np.inf).min(1)
        ok = np.isfinite(kv) & np.isfinite(kc)
        assert (stats[s][10] == (kc - kv)[ok].min()) if ok.any() else np.isnan(stats[s][10])
        assert bs is not None


@pytest.mark.parametrize("npts", [5000, 1001])
def test_gap_centre_of_a_wide_gap_is_the_first_zero_of_the_summed_terms(npts):
    """Through the subnormal numbers the minimum's place hangs on each term's rounding: the point must be the one of the
    DOS summed term by term (the same exponential, on the GPU), gap by gap.  Weights that make no ties."""
    B = _Batch([(1, 4), (3, 6)] * 40, seed=11)
    rng = np.random.default_rng(5)
    sigma, lo, hi = 0.1, -10.0, 10.0
    for s, e in enumerate(B.eig):
        half = rng.uniform(3.4, 4.6, 2) / H2E
        nb = e.shape[1]
        e[:, : nb // 2] = -half[0] - rng.uniform(0.0, 0.02, (len(e), nb // 2))
        e[:, nb // 2:] = half[1] + rng.uniform(0.0, 0.02, (len(e), nb - nb // 2))
        e.sort(axis=1)
        B.w[s] = np.ones(1) if len(e) == 1 else np.array([0.3, 0.34, 0.36])
    B.E, B.kw = _dev(np.concatenate([e.reshape(-1) for e in B.eig]), torch.float64), _dev(np.concatenate(B.w), torch.float64)
    grid, dos, stats = _dos(B, np.zeros(B.n), lo, hi, npts, sigma, 0.0)
    g = torch.as_tensor(grid, device=DEV)
    inside = np.abs(grid) < 2.0
    flat = 0
    for s, e in enumerate(B.eig):
        ref = torch.zeros_like(g)
        for k in range(len(e)):
            sk = torch.zeros_like(g)
            for ev in e[k]:
                t = (g - ev * H2E) * (1.0 / sigma)
                sk = sk + torch.exp(-0.5 * (t * t)) * (1.0 / (sigma * np.sqrt(2.0 * np.pi)))
            ref = ref + float(B.w[s][k]) * sk
        r = np.where(inside, ref.cpu().numpy(), np.inf)
        assert stats[s, 17] == grid[r.argmin()], (s, stats[s, 17], grid[r.argmin()])
        small = inside & (r < 1e-307)
        flat += int(small.any())
        # 2e-11 of the sum, as above, and the last place of each subnormal term
        assert (np.abs(dos[s][small] - r[small]) <= 2e-11 * r[small] + e.size * 4.0 * 4.95e-324).all()
    assert flat > 20
