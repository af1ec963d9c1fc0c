"""Blocked eigensolver (csrc/eigh_panels.cu) on a GB300, against LAPACK and the one-CTA kernel.

Sizes sit at the edges of its panels (32 columns in the factorisations, 16 in the tridiagonalisation), of the
32-wide tiles of the matrix-vector products and of the 128 x 16 tiles of the tensor-core updates; a call mixes
sizes.  The scratch starts as NaN.
"""
import ctypes

import numpy as np
import pytest
import scipy.linalg as sla
import torch

from slakonet_gb300._lib import call, ptr

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _pairs(sizes, seed, real=()):
    rng = np.random.default_rng(seed)
    Hs, Ss = [], []
    for i, n in enumerate(sizes):
        cx = 0.0 if i in real else 1j
        X = rng.standard_normal((n, n)) + cx * rng.standard_normal((n, n))
        Y = (rng.standard_normal((n, n)) + cx * rng.standard_normal((n, n))) * 0.3
        Hs.append(((X + X.conj().T) / 2).astype(np.complex128))
        Ss.append((np.eye(n) + Y @ Y.conj().T / n).astype(np.complex128))
    return Hs, Ss


def _setup(Hs, Ss):
    sizes = np.array([h.shape[0] for h in Hs])
    flat = [np.concatenate([m.T.reshape(-1) for m in ms]) for ms in (Hs, Ss)]
    H, S = (torch.as_tensor(np.stack([f.real, f.imag], 1).reshape(-1), device=DEV) for f in flat)
    off = np.concatenate([[0], np.cumsum(sizes.astype(np.int64) ** 2)[:-1]])
    eo = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int64)
    dev = lambda a: torch.as_tensor(a, device=DEV)   # noqa: E731
    return sizes, H, S, dev(sizes.astype(np.int32)), dev(off), dev(eo), eo


def _panels(Hs, Ss, real=None, slots=None, max_n=None, sms=0):
    sizes, H, S, nv, off, eod, eo = _setup(Hs, Ss)
    slots = np.arange(len(sizes)) if slots is None else np.asarray(slots)
    rl = None if real is None else torch.as_tensor(np.asarray(real, np.int32), device=DEV)
    eig = torch.full((int(sizes.sum()),), -7.0, dtype=torch.float64, device=DEV)
    st = torch.full((len(sizes),), -1, dtype=torch.int32, device=DEV)
    host = np.ascontiguousarray(np.sort(sizes[slots])[::-1].astype(np.int32))
    order = slots[np.argsort(-sizes[slots], kind="stable")]
    prob = torch.as_tensor(order.astype(np.int32), device=DEV)
    if max_n is not None:
        host = np.minimum(host, max_n).astype(np.int32)
    need, at = ctypes.c_int64(0), []
    total = 0
    for n in host:
        at.append(total)
        call("skn_eigh_panels_scratch_bytes", int(n), ctypes.addressof(need))
        total += need.value
    ws = torch.as_tensor(np.array(at, np.int64), device=DEV)
    scratch = torch.full((total // 8,), float("nan"), dtype=torch.float64, device=DEV)
    call("skn_eigh_gen_panels", len(slots), host.ctypes.data, ptr(prob), ptr(ws), ptr(nv), ptr(rl), ptr(off), ptr(eod),
         ptr(H), ptr(S), ptr(eig), ptr(st), 0, ptr(scratch), total, sms, torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize(DEV)
    e = eig.cpu().numpy()
    return [e[o:o + n] for o, n in zip(eo, sizes)], st.cpu().numpy()


def _one_cta(Hs, Ss):
    sizes, H, S, nv, off, eod, eo = _setup(Hs, Ss)
    order = torch.arange(len(sizes), dtype=torch.int32, device=DEV)
    eig = torch.empty(int(sizes.sum()), dtype=torch.float64, device=DEV)
    st = torch.empty(len(sizes), dtype=torch.int32, device=DEV)
    ctr = torch.zeros(2, dtype=torch.int32, device=DEV)
    call("skn_eigh_gen_batched", len(sizes), ptr(nv), ptr(off), ptr(eod), ptr(order), ptr(H), ptr(S), ptr(eig), ptr(st),
         ptr(ctr), int(sizes.max()), torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize(DEV)
    e = eig.cpu().numpy()
    return [e[o:o + n] for o, n in zip(eo, sizes)]


def _bound(n, ref):
    """Backward error of the reductions, a small multiple of n eps, times the spectrum's scale over the smallest
    eigenvalue of S (one or more here)."""
    return 20.0 * n * 2.2e-16 * max(1.0, float(np.abs(ref).max()))


@pytest.mark.parametrize("sizes", [(1, 2, 17, 32), (33, 34, 48, 49, 50, 64), (65, 80, 81, 82, 96), (97, 113, 128),
                                   (129, 145, 160), (257, 272, 288), (385, 400, 401, 402, 416), (513, 534, 544), (1000,), (1300,),
                                   (3, 40, 97, 128, 129, 210, 256, 300)])
def test_blocked_solver_agrees_with_lapack(sizes):
    Hs, Ss = _pairs(sizes, seed=sum(sizes))
    got, st = _panels(Hs, Ss)
    assert (st == 0).all(), st
    ref = [sla.eigh(h, s, eigvals_only=True) for h, s in zip(Hs, Ss)]
    one = _one_cta(Hs, Ss)
    for n, a, r, o in zip(sizes, got, ref, one):
        print(f"n = {n}: vs LAPACK {np.abs(a - r).max():.1e}, one-CTA kernel vs LAPACK {np.abs(o - r).max():.1e}")
    for n, a, r in zip(sizes, got, ref):
        assert np.abs(a - r).max() <= _bound(n, r), n


def test_real_problems_in_a_mixed_call():
    sizes = (97, 128, 110, 128)
    Hs, Ss = _pairs(sizes, seed=4, real=(1, 2))
    plain, _ = _panels(Hs, Ss)
    got, st = _panels(Hs, Ss, real=[0, 1, 1, 0])
    assert (st == 0).all()
    for n, a, b, h, s in zip(sizes, got, plain, Hs, Ss):
        r = sla.eigh(h, s, eigvals_only=True)
        assert np.abs(a - r).max() <= _bound(n, r) and np.abs(b - r).max() <= _bound(n, r)


@pytest.mark.parametrize("sizes", [(150, 129, 160), (300, 289, 320)])
def test_results_do_not_depend_on_the_group(sizes):
    """Alone a problem gets many CTAs (a grid team, or a cluster where fewer SMs are planned for, resident in shared
    memory); among 200 it gets one, streamed."""
    Hs, Ss = _pairs(sizes, seed=9)
    many, _ = _panels(Hs * 70, Ss * 70, slots=np.random.default_rng(1).permutation(210))
    for i in range(3):
        for sms in (0, 20, 8, 2, 1):
            alone, st = _panels([Hs[i]], [Ss[i]], sms=sms)
            assert st[0] == 0
            for q in range(0, 210, 21):
                assert np.array_equal(alone[0], many[q + i]), (i, sms)


def test_indefinite_overlap_and_zero_rows_and_other_sizes():
    sizes = (100, 120, 128, 150)
    Hs, Ss = _pairs(sizes, seed=2)
    Ss[1] = Ss[1] - 2.0 * np.eye(120) * np.abs(Ss[1]).max()
    for m in (Hs[2], Ss[2]):                     # an all-zero row and column counts as a unit diagonal
        m[40, :] = 0.0
        m[:, 40] = 0.0
    got, st = _panels(Hs, Ss, max_n=128)
    assert st.tolist() == [0, 2, 0, 5]           # 150 orbitals in a call for at most 128
    assert np.isnan(got[1]).all() and (got[3] == -7.0).all()
    for i in (0, 2):
        h, s = Hs[i].copy(), Ss[i].copy()
        if i == 2:
            h[40, 40] = s[40, 40] = 1.0
        r = sla.eigh(h, s, eigvals_only=True)
        assert np.abs(got[i] - r).max() <= _bound(sizes[i], r)


def check_scaled_and_graded(n, solve):
    """Powers of two scale exactly, so a scaled pencil's eigenvalues have the plain one's relative error (its vectors have
    the matrix's scale beside entries of at most 1); a graded matrix has eigenvalues far below its norm, each within the
    norm's backward error."""
    Hs, Ss = _pairs((n,), seed=1)
    h, s = Hs[0], Ss[0]
    r = sla.eigh(h, s, eigvals_only=True)
    for a, b in ((1.0, 1.0), (2.0 ** 40, 1.0), (2.0 ** -37, 1.0), (2.0 ** 300, 1.0), (1.0, 2.0 ** 100), (2.0 ** -90, 2.0 ** 90)):
        assert np.abs(solve(h * a, s * b) * (b / a) - r).max() <= _bound(n, r), (a, b)
    d = np.logspace(0, -6, n)
    g = d[:, None] * h * d[None]
    r = sla.eigh(g, s, eigvals_only=True)
    assert np.abs(solve(g, s) - r).max() <= _bound(n, r)


@pytest.mark.parametrize("n", [100, 200, 500])
def test_scaled_and_graded_pencils(n):
    check_scaled_and_graded(n, lambda h, s: _panels([h], [s])[0][0])


def test_scaled_and_graded_pencils_on_the_one_cta_kernel():
    check_scaled_and_graded(100, lambda h, s: _one_cta([h], [s])[0])
