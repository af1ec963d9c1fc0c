"""Eigenvector stage (csrc/eigvec.cu) behind both eigensolvers, and the projectors of the adjoint, on a GB300.

Sizes sit at the edges of the 32-column tiles, of the two solvers (96/97) and of the shared-memory tile (405
rows fit); a call mixes sizes.
"""
import ctypes

import numpy as np
import pytest
import torch

from slakonet_gb300._lib import SKN_OK, call, load, ptr
from test_gpu_panels import _pairs, _setup

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 2.2e-16


def _vectors(Hs, Ss, real=None, fill=float("nan"), one_cta_scratch=False):
    sizes, H, S, nv, off, eod, eo = _setup(Hs, Ss)
    count, most = len(sizes), int(sizes.max())
    rl = None if real is None else torch.as_tensor(np.asarray(real, np.int32), device=DEV)
    eig = torch.empty(int(sizes.sum()), dtype=torch.float64, device=DEV)
    tri = torch.full((4 * int(sizes.sum()),), fill, dtype=torch.float64, device=DEV)
    st = torch.full((count,), -1, dtype=torch.int32, device=DEV)
    stream = torch.cuda.current_stream(DEV).cuda_stream
    order = np.argsort(-sizes, kind="stable").astype(np.int32)
    prob = torch.as_tensor(order, device=DEV)
    if most <= 96:
        call("skn_eigh_gen_small", count, most, ptr(prob), ptr(nv), ptr(rl), ptr(off), ptr(eod), ptr(H), ptr(S), ptr(eig),
             ptr(st), ptr(tri), stream)
    else:
        host = np.ascontiguousarray(sizes[order].astype(np.int32))
        need, at, total = ctypes.c_int64(0), [], 0
        for n in host:
            at.append(total)
            call("skn_eigh_panels_scratch_bytes", int(n), ctypes.addressof(need))
            total += need.value
        ws = torch.as_tensor(np.array(at, np.int64), device=DEV)
        scr = torch.full((total // 8,), fill, dtype=torch.float64, device=DEV)
        call("skn_eigh_gen_panels", count, host.ctypes.data, ptr(prob), ptr(ws), ptr(nv), ptr(rl), ptr(off), ptr(eod),
             ptr(H), ptr(S), ptr(eig), ptr(st), ptr(tri), ptr(scr), total, 0, stream)
    need = ctypes.c_int64(0)
    call("skn_eigvec_scratch_bytes", 1 if one_cta_scratch else count, most, ctypes.addressof(need))
    scratch = torch.full((need.value // 8,), fill, dtype=torch.float64, device=DEV)
    vec = torch.full_like(H, fill)
    ctr = torch.full((1,), 7, dtype=torch.int32, device=DEV)
    args = [count, most, ptr(prob), ptr(nv), ptr(rl), ptr(off), ptr(eod), ptr(H), ptr(S), ptr(eig), ptr(tri), ptr(st),
            ptr(vec), ptr(scratch), need.value, ptr(ctr), stream]
    assert load().skn_eigvec(*args[:14], 8, *args[15:]) != SKN_OK          # less than one CTA's part
    call("skn_eigvec", *args)
    torch.cuda.synchronize(DEV)
    v = torch.view_as_complex(vec.view(-1, 2)).cpu().numpy()
    e, o = eig.cpu().numpy(), off.cpu().numpy()
    return [(e[a:a + n], v[b:b + n * n].reshape(n, n)) for a, b, n in zip(eo, o, sizes)], st.cpu().numpy()


def _check(h, s, e, C):
    """Residual: a backward error of a small multiple of n eps times the norms.  Orthonormality: the vectors of two
    eigenvalues are orthogonal to that error over their distance (no smaller than what is re-orthogonalised)."""
    n, scale = len(e), max(1.0, np.abs(e).max())
    norm = scale * max(1.0, np.linalg.norm(s, 2))
    r = np.abs(h @ C - (s @ C) * e).max()
    assert r <= 50.0 * n * EPS * norm, (n, r)
    gap = max(np.diff(e).min(), 1e-9 * scale) if n > 1 else scale
    o = np.abs(C.conj().T @ s @ C - np.eye(n)).max()
    assert o <= 50.0 * n * EPS * (1.0 + norm / gap), (n, o, gap)


@pytest.mark.parametrize("sizes", [(1, 2, 3, 16, 31, 32, 33), (63, 64, 65, 95, 96), (97, 1, 128, 129, 161, 5),
                                   (404, 405, 406), (600,)])
@pytest.mark.parametrize("real", [False, True])
def test_vectors_solve_the_pencil(sizes, real):
    Hs, Ss = _pairs(sizes, seed=len(sizes), real=range(len(sizes)) if real else ())
    got, st = _vectors(Hs, Ss, real=[1] * len(sizes) if real else None)
    assert (st == 0).all(), st
    for h, s, (e, C) in zip(Hs, Ss, got):
        _check(h, s, e, C)


def test_vectors_do_not_depend_on_the_call():
    sizes = (97, 33, 128, 64)
    Hs, Ss = _pairs(sizes, seed=6)
    together, _ = _vectors(Hs, Ss, fill=0.0, one_cta_scratch=True)
    for i in (0, 2):
        alone, st = _vectors([Hs[i]], [Ss[i]])
        assert st[0] == 0 and np.array_equal(alone[0][1], together[i][1])


def test_indefinite_overlap_gives_nan_vectors_there_alone():
    sizes = (40, 20, 30)
    Hs, Ss = _pairs(sizes, seed=3)
    Ss[1] = Ss[1] - 2.0 * np.eye(20) * np.abs(Ss[1]).max()
    got, st = _vectors(Hs, Ss)
    assert st.tolist() == [0, 2, 0] and np.isnan(got[1][1].real).all()
    for i in (0, 2):
        _check(Hs[i], Ss[i], *got[i])


@pytest.mark.parametrize("sizes", [(1, 15, 16, 17, 31, 32), (33, 64, 65), (100, 7, 161)])
def test_adjoint_projectors(sizes):
    """Sums of n products: n eps of the sum of their magnitudes.  Bands of zero weight at both ends; problem 1 failed."""
    rng = np.random.default_rng(len(sizes))
    sizes = np.array(sizes)
    C = [rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) for n in sizes]
    e, g = ([rng.standard_normal(n) for n in sizes] for _ in range(2))
    for x in g:
        x[: len(x) // 3] = 0.0
        x[len(x) - len(x) // 4:] = 0.0
    flat = np.concatenate([c.reshape(-1) for c in C])
    dev = lambda a, t=np.float64: torch.as_tensor(np.asarray(a, t), device=DEV)   # noqa: E731
    vec = dev(np.stack([flat.real, flat.imag], 1).reshape(-1))
    off = np.concatenate([[0], np.cumsum(sizes ** 2)[:-1]])
    eo = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    st = np.zeros(len(sizes))
    st[1] = 2
    G, F = torch.full_like(vec, float("nan")), torch.full_like(vec, float("nan"))
    keep = [dev(sizes, np.int32), dev(off, np.int64), dev(eo, np.int64), dev(np.concatenate(e)), dev(np.concatenate(g)),
            dev(st, np.int32)]
    call("skn_adj_projectors", len(sizes), *(ptr(t) for t in keep[:3]), ptr(vec), *(ptr(t) for t in keep[3:]), ptr(G), ptr(F),
         torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize(DEV)
    for M, w in ((G, g), (F, [a * b for a, b in zip(g, e)])):
        m = torch.view_as_complex(M.view(-1, 2)).cpu().numpy()
        for q, n in enumerate(sizes):
            out = m[off[q]: off[q] + n * n].reshape(n, n)
            if q == 1:
                assert (out == 0).all()
                continue
            ref = (C[q] * w[q]) @ C[q].conj().T                       # row b, column a
            mag = (np.abs(C[q]) * np.abs(w[q])) @ np.abs(C[q]).T
            assert (np.abs(out - ref) <= 4.0 * (n + 4) * EPS * mag).all()
