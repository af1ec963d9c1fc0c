"""A captured graph stays valid while its batch is solved in other ways (needs a GB300): the graph reads the batch's problem
lists and scratch offsets, whatever later solves with eigenvectors or another policy plan for themselves."""
import numpy as np
import pytest
import torch

from slakonet_gb300 import autotune as AT, engine as E, synthetic as syn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _same(a, b):
    return bool(((a == b) | (torch.isnan(a) & torch.isnan(b))).all())


def test_replay_after_a_solve_with_vectors_and_another_policy():
    rng = np.random.default_rng(5)
    sts = []
    for n in (2, 7, 14, 30):                                  # small groups and two panel classes
        st = syn.random_structure(rng, n, zmax=30)
        st["kpoints"] = rng.uniform(-0.5, 0.5, (5, 3))
        sts.append(st)
    zs = sorted({int(z) for st in sts for z in st["numbers"]})
    sd = syn.default_shell_dict()
    ts = E.TableSet.from_synthetic(syn.make_tables(zs, sd, seed=4), sd, DEV)
    eng = E.Engine(ts)
    plan = E.plan_batch(sts, ts)
    assert plan.max_n > 128
    db = E.DeviceBatch(plan, DEV)
    kw = dict(dos_range=(-20.0, 10.0), dos_points=500, dos_window=9.0)
    cap = E.CapturedPath(eng, db, **kw)
    ref = {k: getattr(cap.result, k).clone() for k in ("eig", "dos", "stats", "mu")}
    res = eng.execute(db, vectors=True, **kw)
    E.Engine(ts, tuning=AT.Tuning.one_cta()).execute(db, **kw)
    torch.cuda.synchronize()
    junk = [torch.full((n,), 1 << 20, dtype=torch.int32, device=DEV) for n in (64, 128, 256, 512, 1024, 4096) * 20]
    out = cap.replay()
    torch.cuda.synchronize()
    assert junk and res.eig.shape == ref["eig"].shape
    for k, v in ref.items():
        assert _same(getattr(out, k), v), k
