"""Infinities and NaNs in a pencil (needs a GB300): every eigenvalue of that problem is NaN, on each eigensolver, and the other
problems of the call are what they are without it."""
import numpy as np
import pytest
import torch

from slakonet_gb300._lib import call, ptr
from test_gpu_panels import DEV, _one_cta, _pairs, _panels, _setup
from test_gpu_small import _small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 16, 33, 64, 65, 100, 130, 300])
@pytest.mark.parametrize("place", ["corner", "diagonal", "last"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_no_finite_eigenvalue_comes_out(n, place, value):
    Hs, Ss = _pairs((n, max(1, n - 1)), seed=n)
    i, j = {"corner": (n - 1, 0), "diagonal": (n // 2, n // 2), "last": (n - 1, n - 1)}[place]
    solve = _small if n <= 64 else _panels
    plain, _ = solve(Hs, Ss)
    bad = [Hs[0].copy(), Hs[1]]
    bad[0][i, j] = value
    got, st = solve(bad, Ss)
    assert np.isnan(got[0]).all() and np.array_equal(got[1], plain[1]) and st[1] == 0
    one = _one_cta(bad, Ss)
    assert np.isnan(one[0]).all() and np.isfinite(one[1]).all()


def test_the_device_wide_and_the_cluster_path():
    import ctypes
    from test_gpu_wide import _pairs as pairs, _wide
    Hs, Ss = pairs(150, 2, seed=3)
    Hs[0][149, 7] = np.inf
    got, st = _wide(Hs, Ss)
    assert np.isnan(got[0]).all() and np.isfinite(got[1]).all() and st[1] == 0
    sizes, H, S, nv, off, eod, _ = _setup(Hs, Ss)
    order = torch.arange(2, dtype=torch.int32, device=DEV)
    eig = torch.zeros(300, dtype=torch.float64, device=DEV)
    stt, ctr = torch.zeros(2, dtype=torch.int32, device=DEV), torch.zeros(2, dtype=torch.int32, device=DEV)
    need = ctypes.c_int64(0)
    call("skn_eigh_large_scratch_bytes", 2, 150, 4, ctypes.addressof(need))
    scr = torch.zeros(need.value // 8, dtype=torch.float64, device=DEV)
    call("skn_eigh_gen_large", 2, ptr(nv), ptr(off), ptr(eod), ptr(order), ptr(H), ptr(S), ptr(eig), ptr(stt), ptr(ctr),
         ptr(scr), need.value, 150, 4, torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize(DEV)
    e = eig.cpu().numpy()
    assert np.isnan(e[:150]).all() and np.isfinite(e[150:]).all()
