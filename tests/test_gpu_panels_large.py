"""Blocked eigensolver and its vectors on a GB300 above 1024 rows, up to the bound of 2048 orbitals: streamed columns of more
rows than the threads hold at once, calls that mix sizes, plans by rounds with two CTAs to an SM."""
import numpy as np
import pytest
import scipy.linalg as sla

from test_gpu_eigvec_stage import _check, _vectors
from test_gpu_panels import _bound, _pairs, _panels

pytestmark = pytest.mark.gpu


def test_streamed_columns_above_1024_rows_give_the_resident_bits():
    Hs, Ss = _pairs((1300,), seed=5)
    resident, st = _panels(Hs, Ss)
    streamed, st1 = _panels(Hs, Ss, sms=1)
    assert st[0] == 0 and st1[0] == 0 and np.array_equal(resident[0], streamed[0])
    r = sla.eigh(Hs[0], Ss[0], eigvals_only=True)
    assert np.abs(resident[0] - r).max() <= _bound(1300, r)


@pytest.mark.parametrize("sizes", [(2048, 1100, 1025), (2047, 1660, 1633)])
def test_mixed_calls_up_to_the_bound(sizes):
    Hs, Ss = _pairs(sizes, seed=sum(sizes), real=(2,))
    together, st = _panels(Hs, Ss, real=[0, 0, 1])                   # streamed: by rounds, with the GPU to itself
    beside, st1 = _panels(Hs, Ss, real=[0, 0, 1], sms=1)             # and one CTA each
    assert (st == 0).all() and (st1 == 0).all()
    for i, n in enumerate(sizes):
        assert np.array_equal(together[i], beside[i]), n
        alone, st = _panels([Hs[i]], [Ss[i]], real=[int(i == 2)])
        assert st[0] == 0 and np.array_equal(alone[0], together[i]), n
    i = 0 if sizes[0] == 2048 else 1
    r = sla.eigh(Hs[i], Ss[i], eigvals_only=True)
    assert np.abs(together[i] - r).max() <= _bound(sizes[i], r)


@pytest.mark.parametrize("sizes", [(1300, 1025), (2048,)])
def test_vectors_up_to_the_bound(sizes):
    Hs, Ss = _pairs(sizes, seed=7)
    got, st = _vectors(Hs, Ss)
    assert (st == 0).all()
    for h, s, (e, C) in zip(Hs, Ss, got):
        _check(h, s, e, C)
