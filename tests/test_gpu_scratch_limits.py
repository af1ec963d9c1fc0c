"""A batch that leaves little room for scratch is still solved (needs a GB300): with the allocator limited to what the rest
of the path holds and a part of the scratch, the panel groups go through in smaller parts, to the same bits; with no room
at all, values come from the one-CTA kernel, which needs no scratch."""
import gc

import numpy as np
import pytest
import torch

from slakonet_gb300 import engine as E, synthetic as syn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MIB = 1 << 20


@pytest.fixture
def batch(monkeypatch):
    monkeypatch.setattr(E, "PANELS_SCRATCH", 1024 * MIB)        # so that a small batch meets the limits; parts of 64 MB
    rng = np.random.default_rng(8)
    sts = []
    for n in (9, 12, 16, 20):
        st = syn.random_structure(rng, n, zmax=30)
        st["kpoints"] = rng.uniform(-0.5, 0.5, (80, 3))
        sts.append(st)
    zs = sorted({int(z) for st in sts for z in st["numbers"]})
    sd = syn.default_shell_dict()
    ts = E.TableSet.from_synthetic(syn.make_tables(zs, sd, seed=4), sd, DEV)
    yield ts, E.DeviceBatch(E.plan_batch(sts, ts), DEV)
    torch.cuda.set_per_process_memory_fraction(1.0)
    torch.cuda.empty_cache()


def _clean():
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()


def _limit(nbytes):
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction(nbytes / total)


@pytest.mark.parametrize("vectors", [False, True])
def test_less_room_gives_the_same_results(batch, vectors):
    ts, db = batch
    tried = []

    class Engine(E.Engine):
        def _scratch(self, groups, vec, vec_budget):
            tried.append(sum(max(p[3] for p in g.parts) for g in groups if g.parts))
            return super()._scratch(groups, vec, vec_budget)
    eng = Engine(ts)
    kw = dict(dos_points=200, vectors=vectors)
    eng.execute(db, **kw)
    _clean()
    ref = eng.execute(db, **kw)
    full = tried[-1]
    assert full > 256 * MIB and len(tried) == 2
    peak = torch.cuda.max_memory_allocated()
    host = {k: getattr(ref, k).cpu() for k in ("eig", "dos", "mu") + (("vec",) if vectors else ())}
    status = ref.eig_status.cpu()
    del ref
    _clean()
    tried.clear()
    _limit(peak - full + 160 * MIB)                              # room for the parts, not for all at once
    out = eng.execute(db, **kw)
    assert len(tried) > 1 and tried[-1] < full
    assert torch.equal(out.eig_status.cpu(), status)
    for k, v in host.items():
        assert torch.equal(getattr(out, k).cpu(), v), k


def test_no_room_at_all_still_gives_values(batch):
    ts, db = batch
    eng = E.Engine(ts)
    eng.execute(db, dos_points=200)
    _clean()
    ref = eng.execute(db, dos_points=200)
    peak = torch.cuda.max_memory_allocated()
    full = sum(max(p[3] for p in g.parts) for g in eng._groups(db, False, E.PANELS_SCRATCH) if g.parts)
    eig = ref.eig.cpu()
    del ref
    _clean()
    _limit(peak - full + 40 * MIB)
    out = eng.execute(db, dos_points=200)
    assert (out.eig_status == 0).all()
    assert (False, 0) in {k[:2] for k in db.groups}              # the plan without scratch was made
    d = (out.eig.cpu() - eig).abs().max()
    # two backward-stable solvers of up to 320 orbitals: 2 x 20 n eps of the spectrum's scale
    assert d <= 2 * 20 * 320 * 2.2e-16 * max(1.0, float(eig.abs().max()))
