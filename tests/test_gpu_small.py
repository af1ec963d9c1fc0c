"""Shared-memory eigensolver (csrc/eigh_small.cu) on a GB300, against LAPACK.

Every size from 1 to 96 goes through each of its three thread counts' edges (16, 32, 96); a call mixes sizes.
"""
import numpy as np
import pytest
import scipy.linalg as sla
import torch

from slakonet_gb300._lib import call, ptr
from test_gpu_panels import _bound, _pairs, _setup, check_scaled_and_graded

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _small(Hs, Ss, real=None, max_n=None):
    sizes, H, S, nv, off, eod, eo = _setup(Hs, Ss)
    prob = torch.arange(len(sizes), dtype=torch.int32, device=DEV)
    rl = None if real is None else torch.as_tensor(np.asarray(real, np.int32), device=DEV)
    eig = torch.full((int(sizes.sum()),), -7.0, dtype=torch.float64, device=DEV)
    st = torch.full((len(sizes),), -1, dtype=torch.int32, device=DEV)
    call("skn_eigh_gen_small", len(sizes), int(max_n or sizes.max()), ptr(prob), ptr(nv), ptr(rl), ptr(off), ptr(eod),
         ptr(H), ptr(S), ptr(eig), ptr(st), 0, torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize(DEV)
    e = eig.cpu().numpy()
    return [e[o:o + n] for o, n in zip(eo, sizes)], st.cpu().numpy()


@pytest.mark.parametrize("lo,hi", [(1, 16), (17, 32), (33, 64), (65, 96)])
@pytest.mark.parametrize("real", [False, True])
def test_every_size_agrees_with_lapack(lo, hi, real):
    sizes = tuple(range(lo, hi + 1))
    Hs, Ss = _pairs(sizes, seed=lo, real=range(len(sizes)) if real else ())
    got, st = _small(Hs, Ss, real=[1] * len(sizes) if real else None)
    assert (st == 0).all(), st
    worst = 0.0
    for n, a, h, s in zip(sizes, got, Hs, Ss):
        r = sla.eigh(h, s, eigvals_only=True)
        worst = max(worst, np.abs(a - r).max())
        assert np.abs(a - r).max() <= _bound(n, r), n
    print(f"n = {lo}-{hi}: vs LAPACK {worst:.1e}")


def test_indefinite_overlap_zero_rows_and_capacity():
    sizes = (30, 20, 40, 33)
    Hs, Ss = _pairs(sizes, seed=3)
    Ss[1] = Ss[1] - 2.0 * np.eye(20) * np.abs(Ss[1]).max()
    for m in (Hs[3], Ss[3]):
        m[7, :] = 0.0
        m[:, 7] = 0.0
    got, st = _small(Hs, Ss, max_n=39)
    assert st.tolist() == [0, 2, 5, 0]
    assert np.isnan(got[1]).all() and (got[2] == -7.0).all()
    for i in (0, 3):
        h, s = Hs[i].copy(), Ss[i].copy()
        if i == 3:
            h[7, 7] = s[7, 7] = 1.0
        r = sla.eigh(h, s, eigvals_only=True)
        assert np.abs(got[i] - r).max() <= _bound(sizes[i], r)


def test_results_do_not_depend_on_the_call():
    sizes = (33, 64, 41, 96)
    Hs, Ss = _pairs(sizes, seed=6)
    together, _ = _small(Hs, Ss)
    for i in range(4):
        alone, st = _small([Hs[i]], [Ss[i]])
        assert st[0] == 0 and np.array_equal(alone[0], together[i])


@pytest.mark.parametrize("n", [40, 96])
def test_scaled_and_graded_pencils(n):
    check_scaled_and_graded(n, lambda h, s: _small([h], [s])[0][0])
