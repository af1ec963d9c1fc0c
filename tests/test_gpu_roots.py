"""Pivots and reflectors from reciprocal roots (csrc/eigh_small.cu, eigh_panels.cu) on a GB300, against the square root.

With a reciprocal root within one last place, the Newton step leaves the root within one last place of the rounded one
(the step squares the error and rounds once); a factor's column, scaled by the reciprocal, is within three halves of a last
place of it and a rounding: 2 eps relative; the small kernel's beta is the root of a sum of two squares, two roundings more: 2 eps
(the panel kernel takes the same steps, on entries held relative to their row's largest).  Scales from 2^-400 to 2^400, and values just beside powers of two."""
import ctypes

import numpy as np
import pytest
import torch

from slakonet_gb300._lib import call, ptr
from test_gpu_panels import _setup

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 2.0 ** -52
LD = np.longdouble


def _factor(Hs, Ss, panels):
    """(L in S's lower triangle, tri) as the values kernel leaves them for the vectors."""
    sizes, H, S, nv, off, eod, _ = _setup(Hs, Ss)
    count, n = len(sizes), int(sizes.max())
    prob = torch.arange(count, dtype=torch.int32, device=DEV)
    eig = torch.zeros(int(sizes.sum()), dtype=torch.float64, device=DEV)
    st = torch.zeros(count, dtype=torch.int32, device=DEV)
    tri = torch.zeros(4 * int(sizes.sum()), dtype=torch.float64, device=DEV)
    stream = torch.cuda.current_stream(DEV).cuda_stream
    if panels:
        need = ctypes.c_int64(0)
        call("skn_eigh_panels_scratch_bytes", n, ctypes.addressof(need))
        ws = torch.arange(count, dtype=torch.int64, device=DEV) * need.value
        scr = torch.zeros(count * need.value // 8, dtype=torch.float64, device=DEV)
        host = np.full(count, n, np.int32)
        call("skn_eigh_gen_panels", count, host.ctypes.data, ptr(prob), ptr(ws), ptr(nv), 0, ptr(off), ptr(eod), ptr(H), ptr(S),
             ptr(eig), ptr(st), ptr(tri), ptr(scr), count * need.value, 0, stream)
    else:
        call("skn_eigh_gen_small", count, n, ptr(prob), ptr(nv), 0, ptr(off), ptr(eod), ptr(H), ptr(S), ptr(eig), ptr(st),
             ptr(tri), stream)
    torch.cuda.synchronize(DEV)
    assert (st == 0).all()
    L = torch.view_as_complex(S.view(-1, 2)).cpu().numpy().reshape(count, n, n).transpose(0, 2, 1)
    return L, tri.cpu().numpy().reshape(count, 4 * n)


def _values(count, rng):
    a = rng.uniform(1.0, 4.0, count) * 2.0 ** (2 * rng.integers(-200, 200, count)).astype(float)
    edge = np.array([1.0, 1.0 + EPS, 1.0 - EPS / 2, 2.0, 4.0 - 2 * EPS, 4.0, 4.0 + 4 * EPS, 0.25, 9.0, 3.0])
    a[:len(edge)] = edge
    return a


@pytest.mark.parametrize("panels", [False, True])
def test_pivots_and_columns_of_the_factor(panels):
    rng = np.random.default_rng(1)
    a = _values(2000, rng)
    z = (rng.uniform(0.1, 0.9, 2000) * np.exp(2j * np.pi * rng.uniform(0, 1, 2000))) * a
    Hs, Ss = [], []
    for x, y in zip(a, z):
        Hs.append(np.diag([x, 2.0 * x]).astype(complex))
        Ss.append(np.array([[x, np.conj(y)], [y, 2.0 * x]]))
    L, _ = _factor(Hs, Ss, panels)
    root = np.sqrt(a)
    assert (np.abs(L[:, 0, 0].real - root) <= np.spacing(root)).all()
    want = z.astype(np.clongdouble) / np.sqrt(a.astype(LD))
    for got, ref in ((L[:, 1, 0].real, want.real), (L[:, 1, 0].imag, want.imag)):
        # panels: the column goes through the block's inverse in fixed point, relative to the larger part
        tol = 2 * EPS * (np.abs(want).astype(float) if panels else np.abs(ref).astype(float))
        assert (np.abs((got - ref).astype(float)) <= tol).all()


def test_reflectors():
    rng = np.random.default_rng(2)
    a = np.sqrt(_values(2000, rng))
    z = a * np.exp(2j * np.pi * rng.uniform(0, 1, 2000))
    Hs = [np.array([[1.0, np.conj(y)], [y, 2.0]]) for y in z]
    _, tri = _factor(Hs, [np.eye(2, dtype=complex)] * 2000, False)
    re, im = z.real.astype(LD), z.imag.astype(LD)
    want = np.sqrt(re * re + im * im)
    assert (np.abs((np.abs(tri[:, 2]).astype(LD) - want) / want).astype(float) <= 2 * EPS).all()
