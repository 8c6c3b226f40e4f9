"""The tuning search times what differs: one candidate per row-piece width, the
automatic rule among them, each once.  No GPU: the timing is replaced."""
import pytest

import resvg_gb300 as R
from resvg_gb300 import batch as BT


def test_candidates_are_the_row_widths():
    px = [p for _, p in BT.TUNING_CANDIDATES]
    assert sorted(px) == sorted(set(px)) and 0 in px
    assert {b for b, _ in BT.TUNING_CANDIDATES} == {0}


@pytest.mark.parametrize("fastest", BT.TUNING_CANDIDATES)
def test_each_candidate_is_timed_once_and_the_fastest_installed(native, monkeypatch, fastest):
    import torch
    timed = []

    def fake(R_, torch_, trees, ws, hs, ptrs, stream, reps):
        timed.append(R_.get_tuning())
        return 1.0 if timed[-1] == fastest else 2.0 + len(timed)

    monkeypatch.setattr(BT, "_time_scene", fake)
    monkeypatch.setattr(torch.cuda, "Stream", lambda *a, **k: None)
    saved = R.get_tuning()
    try:
        table, px, timings = BT.autotune_table([None] * 3, [64, 300, 900], [64, 300, 900], [0, 0, 0])
        assert timed == BT.TUNING_CANDIDATES and set(timings["global"]) == set(timed)
        assert px == fastest[1] and R.get_tuning() == (0, px)
        assert R.get_tuning_table() == [tuple(e) for e in table] and table
    finally:
        R.set_tuning_table([])
        R.set_tuning(*saved)
