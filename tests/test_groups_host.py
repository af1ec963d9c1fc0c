"""The eigensolver's groups of a batch (engine.Engine._groups), on the CPU: which call a problem takes, and that what one
solve has planned stays in place, and alive, whatever is solved after it on the same batch (a captured graph reads it)."""
import gc
import types
import weakref

import numpy as np
import pytest
import torch

from slakonet_gb300 import autotune as AT, engine as E, synthetic as syn


def _batch(natoms, nk=2, zmax=20):
    rng = np.random.default_rng(0)
    sts = []
    for n in natoms:
        st = syn.random_structure(rng, n, zmax=zmax)
        st["kpoints"] = rng.uniform(-0.5, 0.5, (nk, 3))
        sts.append(st)
    zs = sorted({int(z) for st in sts for z in st["numbers"]})
    sd = syn.default_shell_dict()
    ts = E.TableSet.from_synthetic(syn.make_tables(zs, sd, seed=1), sd, "cpu")
    return E.DeviceBatch(E.plan_batch(sts, ts), torch.device("cpu"))


def _engine(**kw):
    eng = object.__new__(E.Engine)
    eng.__dict__.update(dict(tuning=None, large_threshold=2048, large_cluster=None, real_path=True, wide_threshold=2048,
                             device=torch.device("cpu")), **kw)
    return eng


@pytest.fixture(autouse=True)
def _sms(monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: types.SimpleNamespace(multi_processor_count=152))


def _arrays(groups):
    for g in groups:
        yield g[1]
        for part in getattr(g, "parts", ()):
            yield part[2]


def test_a_solve_with_vectors_leaves_what_a_captured_graph_reads():
    db = _batch((3, 8, 20, 40))
    eng = _engine()
    first = [weakref.ref(t) for t in _arrays(eng._groups(db))]
    values = [r().clone() for r in first]
    assert len(first) > 4
    eng._groups(db, True)                                     # vectors, then other policies, on the same batch
    for n in range(8):
        eng.tuning = AT.Tuning({64: ["", "_blk"][n & 1], 128: "_blk"})
        eng._groups(db)
        gc.collect()
    assert all(r() is not None and torch.equal(r(), v) for r, v in zip(first, values))
    eng.tuning = None
    assert [id(t) for t in _arrays(eng._groups(db))] == [id(r()) for r in first]
