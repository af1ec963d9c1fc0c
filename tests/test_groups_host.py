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


def test_scratch_of_all_groups_stays_within_the_budget():
    gib = 1 << 30
    assert E.scratch_shares([3, 1, 2], [1, 1, 1], 10) == [3, 1, 2]
    assert E.scratch_shares([8 * gib, gib, 20 * gib], [1, 1, 1], 16 * gib) == [7.5 * gib, gib, 7.5 * gib]
    assert E.scratch_shares([8, 9], [5, 6], 0) == [5, 6]       # never less than one problem's
    assert E.scratch_shares([], [], 5) == []
    rng = np.random.default_rng(1)
    for _ in range(50):
        need = [int(x) for x in rng.integers(1, 1 << 34, rng.integers(1, 32))]
        least = [min(n, 50 << 20) for n in need]
        got = E.scratch_shares(need, least, 16 * gib)
        assert sum(got) <= 16 * gib + sum(least) and all(a <= b for a, b in zip(got, need))


@pytest.mark.parametrize("budget", [E.PANELS_SCRATCH, 64 << 20, 4 << 20])
@pytest.mark.parametrize("vectors", [False, True])
def test_parts_cover_every_problem_once_within_their_scratch(budget, vectors):
    db = _batch((8, 12, 20, 40, 64), nk=20)
    groups = _engine()._groups(db, vectors, budget)
    seen = np.concatenate([g.order.numpy() for g in groups])
    assert sorted(seen) == list(range(len(db.plan.prob_n)))
    held = 0
    for g in groups:
        assert bool(g.parts) == (g.kind[0] == "panels")
        at = 0
        for first, last, off, nbytes, sizes in g.parts:
            assert first == at and np.array_equal(sizes, db.plan.prob_n[g.order.numpy()[first:last]])
            per = np.array([E.panels_scratch_bytes(n) for n in sizes])
            assert off[0] == 0 and np.array_equal(off.numpy(), np.cumsum(per) - per) and nbytes == per.sum()
            at = last
        assert not g.parts or at == g.count
        held += max((p[3] for p in g.parts), default=0)
    least = sum(E.panels_scratch_bytes(g.max_n) for g in groups if g.parts)
    assert held <= max(budget, least)


def test_without_scratch_values_take_the_one_cta_kernel():
    db = _batch((2, 12, 40))
    kinds = {g.kind for g in _engine()._groups(db, False, 0)}
    assert not any(k[0] == "panels" for k in kinds if isinstance(k, tuple))
    assert {"_blk"} & kinds or {"_real_blk"} & kinds
    assert any(g.parts for g in _engine()._groups(db, True, 0))        # vectors: one problem at a time


def _routes(sizes, tuning=None, **kw):
    """{orbitals: kind of its group} of a stub batch with two problems of each size."""
    n = np.repeat(np.array(sorted(sizes, reverse=True), np.int32), 2)
    plan = types.SimpleNamespace(prob_n=n, nb=np.unique(n), order=np.arange(len(n)), prob_real=None)
    db = types.SimpleNamespace(plan=plan, groups={}, order=torch.arange(len(n), dtype=torch.int32))
    out = {}
    for g in _engine(tuning=tuning, **kw)._groups(db):
        out.update({int(n[p]): g.kind for p in g.order.numpy()})
    return out


SIZES = (10, 60, 432, 1500, 3000)
AUTO_ROUTES = {10: ("small", 16), 60: ("small", 64), 432: ("panels", 7), 1500: ("panels", 24), 3000: ("wide", 3000, 0)}


def test_what_was_not_tuned_keeps_the_default_route():
    assert _routes(SIZES) == AUTO_ROUTES
    assert _routes(SIZES, AT.Tuning({})) == AUTO_ROUTES
    assert _routes(SIZES, AT.Tuning({16: "_t64"})) == {**AUTO_ROUTES, 10: "_t64"}
    assert AT.Tuning({16: "_t64"}).policy_for(9000) == AT.AUTO


def test_one_cta_problems_above_1024_orbitals_go_to_the_device_wide_or_the_cluster_path():
    one = AT.Tuning.one_cta()
    assert _routes(SIZES, one) == {10: "", 60: "", 432: "_blk", 1500: ("wide", 1500, 0), 3000: ("wide", 3000, 0)}
    assert _routes(SIZES, one, wide_threshold=None) == {10: "", 60: "", 432: "_blk", 1500: 4, 3000: 8}
    assert _routes(SIZES, one, wide_threshold=None, large_threshold=None) == {10: "", 60: "", 432: "_blk", 1500: "_blk", 3000: 8}
    assert _routes(SIZES, None, wide_threshold=400)[432] == ("wide", 432, 0)
    # the cluster path between its threshold and 1024 orbitals, where the device-wide one is on
    mid = SIZES + (800,)
    assert _routes(mid, None, large_threshold=600) == {**AUTO_ROUTES, 800: 4, 1500: ("wide", 1500, 0)}
    assert _routes(mid, None, large_threshold=600, wide_threshold=None) == {**AUTO_ROUTES, 800: 4, 1500: 4, 3000: 8}


def test_the_autotuner_times_the_default_route_too(monkeypatch, tmp_path):
    asked = []

    def timed(suffix, n, count, device, reps=2):
        asked.append((suffix, n))
        return {AT.AUTO: 1.0, "_blk": 0.5 if n == 512 else 2.0}.get(suffix, 3.0)
    monkeypatch.setattr(AT, "time_shape", timed)
    monkeypatch.setattr(AT, "_cache_key", lambda d: "k")
    monkeypatch.setattr(AT._lib, "load", lambda: None)
    tun = AT.autotune("cpu", cache=str(tmp_path / "t.json"), buckets=[64, 512])
    assert tun.choice == {64: AT.AUTO, 512: "_blk"} and {s for s, _ in asked} == {AT.AUTO, *AT.SHAPES}
    assert AT.autotune("cpu", cache=str(tmp_path / "t.json"), buckets=[64, 512]).choice == tun.choice


def test_a_refused_launch_leaves_no_side_stream_unjoined(monkeypatch):
    """The calls of a solve run on side streams and share its buffers: also when one of them is refused, what was launched
    before it is waited for on the solve's own stream."""
    import contextlib

    class Stream:
        cuda_stream = 0

        def __init__(self):
            self.waits = []

        def wait_event(self, ev):
            self.waits.append(ev)

    class Event:
        def record(self, stream=None):
            self.stream = stream
    main, sides = Stream(), [Stream() for _ in range(8)]
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: main)
    monkeypatch.setattr(torch.cuda, "stream", lambda st: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "Event", Event)
    eng = _engine(launches=0, wide_tc=True)
    eng._side_streams = lambda k: sides
    calls = []

    def call(name, *args):
        calls.append(name)
        if len(calls) == 3:
            raise E._lib.SknError("refused")
    eng._call = call
    db = _batch((2, 8, 20, 40))
    assert len(eng._groups(db)) >= 4
    t = torch.zeros(1, dtype=torch.float64)
    with pytest.raises(E._lib.SknError):
        eng._eig_values(db, t, t, t, torch.zeros(1, dtype=torch.int32), 0)
    assert [ev.stream for ev in main.waits] == sides[:3]
