"""Admission counts what a request's panel eigensolves hold, and no more than one solve ever holds."""
from slakonet_gb300 import engine as E, serving as SV


def test_admission_counts_the_panel_scratch_up_to_a_solves_budget():
    base = SV.request_bytes(200, 5, 1000)
    per = E.panels_scratch_bytes(200)
    assert SV.request_bytes(200, 5, 1000, panels=True) == base + 5 * per
    nk = 10 * E.PANELS_SCRATCH // per
    assert SV.request_bytes(200, nk, 1000, panels=True) == SV.request_bytes(200, nk, 1000) + E.PANELS_SCRATCH
    for n in (E.SMALL_MAX_N, E.PANELS_MAX_N + 1):
        assert SV.request_bytes(n, 5, 1000, panels=True) == SV.request_bytes(n, 5, 1000)
    for n, ratio in ((65, 11.6), (128, 3.3), (492, 0.85)):
        assert abs(E.panels_scratch_bytes(n) / (32 * n * n) - ratio) < 0.06 * ratio
