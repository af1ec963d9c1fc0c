"""Bounded waits of the device-wide eigensolver's tensor-core updates on a GB300: one that runs out (a limit of no polls)
marks the problem SKN_ERR_CUDA and its eigenvalues are NaN; the next call on the same device works."""
import ctypes

import numpy as np
import pytest
import torch

from slakonet_gb300._lib import SKN_ERR_CUDA, call, ptr
from test_gpu_wide import DEV, _pack, _pairs
from test_gpu_wide_tc import _wide_tc

pytestmark = pytest.mark.gpu


def _limited(Hs, Ss, real, polls):
    n, count = Hs[0].shape[0], len(Hs)
    nv = torch.full((count,), n, dtype=torch.int32, device=DEV)
    off = torch.arange(count, dtype=torch.int64, device=DEV) * n * n
    eo = torch.arange(count, dtype=torch.int64, device=DEV) * n
    prob = torch.arange(count, dtype=torch.int32, device=DEV)
    H, S = _pack(Hs), _pack(Ss)
    eig = torch.full((count * n,), -7.0, dtype=torch.float64, device=DEV)
    st = torch.full((count,), -1, dtype=torch.int32, device=DEV)
    need = ctypes.c_int64(0)
    call("skn_eigh_wide_scratch_bytes", count, n, ctypes.addressof(need))
    scratch = torch.zeros(need.value // 8, dtype=torch.float64, device=DEV)
    call("skn_eigh_gen_wide_tc_limits", count, n, ptr(prob), ptr(nv), ptr(off), ptr(eo), ptr(H), ptr(S), ptr(eig),
         ptr(st), ptr(scratch), need.value, int(real), polls, torch.cuda.current_stream(DEV).cuda_stream)
    torch.cuda.synchronize(DEV)
    return eig.cpu().numpy().reshape(count, n), st.cpu().numpy()


@pytest.mark.parametrize("real", [False, True])
def test_a_wait_that_runs_out_is_reported_and_leaves_nan(real):
    Hs, Ss = _pairs(600, 2, seed=9, real=real)
    got, st = _limited(Hs, Ss, real, 0)
    assert (st == SKN_ERR_CUDA).all() and np.isnan(got).all()
    plain, _ = _wide_tc(Hs, Ss, real=real)
    got, st = _limited(Hs, Ss, real, 1 << 30)
    assert (st == 0).all() and np.array_equal(got, plain)
