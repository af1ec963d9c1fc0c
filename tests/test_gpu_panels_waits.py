"""Bounded waits of the panel eigensolver on a GB300: a wait that runs out (a limit of no polls) marks
the problem SKN_ERR_CUDA, and its eigenvalues and vectors are NaN, not what the buffer held; a limit long enough changes
nothing.  The kernels return and the next call on the same buffers works."""
import ctypes

import numpy as np
import pytest
import torch

from slakonet_gb300._lib import SKN_ERR_CUDA, call, ptr
from test_gpu_panels import _pairs, _panels, _setup

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LONG = 1 << 30


def _limited(Hs, Ss, polls, sms=0, vectors=False):
    sizes, H, S, nv, off, eod, eo = _setup(Hs, Ss)
    order = np.argsort(-sizes, kind="stable")
    host = np.ascontiguousarray(sizes[order].astype(np.int32))
    prob = torch.as_tensor(order.astype(np.int32), device=DEV)
    need, at, total = ctypes.c_int64(0), [], 0
    for n in host:
        at.append(total)
        call("skn_eigh_panels_scratch_bytes", int(n), ctypes.addressof(need))
        total += need.value
    ws = torch.as_tensor(np.array(at, np.int64), device=DEV)
    scratch = torch.zeros(total // 8, dtype=torch.float64, device=DEV)
    eig = torch.full((int(sizes.sum()),), -7.0, dtype=torch.float64, device=DEV)
    st = torch.full((len(sizes),), -1, dtype=torch.int32, device=DEV)
    tri = torch.zeros(4 * int(sizes.sum()), dtype=torch.float64, device=DEV) if vectors else None
    lim = np.array(polls, np.int32)
    stream = torch.cuda.current_stream(DEV).cuda_stream
    call("skn_eigh_gen_panels_limits", len(sizes), host.ctypes.data, ptr(prob), ptr(ws), ptr(nv), 0, ptr(off), ptr(eod),
         ptr(H), ptr(S), ptr(eig), ptr(st), ptr(tri), ptr(scratch), total, sms, lim.ctypes.data, stream)
    vec = None
    if vectors:
        call("skn_eigvec_scratch_bytes", len(sizes), int(sizes.max()), ctypes.addressof(need))
        vs = torch.zeros(need.value // 8, dtype=torch.float64, device=DEV)
        vec, ctr = torch.zeros_like(H), torch.zeros(1, dtype=torch.int32, device=DEV)
        call("skn_eigvec", len(sizes), int(sizes.max()), ptr(prob), ptr(nv), 0, ptr(off), ptr(eod), ptr(H), ptr(S), ptr(eig),
             ptr(tri), ptr(st), ptr(vec), ptr(vs), need.value, ptr(ctr), stream)
    torch.cuda.synchronize(DEV)
    e = eig.cpu().numpy()
    return [e[o:o + n] for o, n in zip(eo, sizes)], st.cpu().numpy(), vec


# no polls: the solves' wait, the updates', a grid team's (300 orbitals alone: 55 tiles, as many CTAs)
@pytest.mark.parametrize("sizes,polls", [((100, 80), (0, LONG, LONG)), ((100, 80), (LONG, 0, LONG)),
                                         ((300,), (LONG, LONG, 0))])
def test_a_wait_that_runs_out_is_reported_and_leaves_nan(sizes, polls):
    Hs, Ss = _pairs(sizes, seed=3)
    got, st, vec = _limited(Hs, Ss, polls, vectors=True)
    assert (st == SKN_ERR_CUDA).all(), st
    assert all(np.isnan(e).all() for e in got)
    assert torch.isnan(vec.view(-1, 2)[:, 0]).all()
    plain, _ = _panels(Hs, Ss)                               # and the context is as usable as before
    again, st, _ = _limited(Hs, Ss, (LONG, LONG, LONG))
    assert (st == 0).all() and all(np.array_equal(a, b) for a, b in zip(plain, again))


def test_a_clustered_team_has_no_wait_that_can_run_out():
    Hs, Ss = _pairs((300,), seed=3)
    plain, _ = _panels(Hs, Ss)
    got, st, _ = _limited(Hs, Ss, (LONG, LONG, 0), sms=8)     # a cluster of 8: the hardware's barrier
    assert st[0] == 0 and np.array_equal(plain[0], got[0])
