"""Batches in which some pairs are filled lane per group and others by one warp per
group (two queues, two launches, kept storage in two forms): short and longer plain
pairs, profiles, an anchored pair, one with a positive gap opening and one wider than
the lanes' span limit, in mixed order. Against the oracle; every call twice (the
second replays the chunk's graph), in one chunk and in several."""
import copy

import pytest

from checks import assert_same_result
from oracle_ffi import oracle_align

_CASES = {}


def _tables(stacking):
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_profile, make_rna
    kw = dict(stacking=1, exp_prob=0.01) if stacking else {}
    tabs = []
    for k, (la, lb) in enumerate([(64, 60), (17, 31), (96, 71), (9, 12), (50, 120), (130, 110)]):
        a = make_rna(la, 500 + k)
        b = make_homolog(a, 3) if k % 2 else make_rna(lb, 550 + k)
        tabs.append(prepare_pair(a.to_pp(stacking=stacking), b.to_pp(stacking=stacking), **kw))
    anchored = [make_rna(70, 81).to_pp(stacking=stacking, anchors="." * 20 + "A" + "." * 30 + "B" + "." * 18),
                make_rna(66, 82).to_pp(stacking=stacking, anchors="." * 22 + "A" + "." * 26 + "B" + "." * 16)]
    tabs.insert(1, prepare_pair(*anchored, **kw))
    opening = copy.copy(tabs[3])
    opening.indel_opening = 30
    tabs.insert(4, opening)
    # the whole band of 24 x 660: a span of 663 columns
    tabs.append(prepare_pair(make_rna(24, 83).to_pp(stacking=stacking), make_rna(660, 84).to_pp(stacking=stacking),
                             min_trace_probability=0.0, **kw))
    if not stacking:
        tabs.insert(6, prepare_pair(make_profile(60, 5).to_pp(), make_profile(52, 6).to_pp()))
    return tabs


MODES = {"global": dict(), "stacking": dict(), "normalized": dict(sequ_local=True, normalized=50),
         "free_endgaps": dict(free_endgaps="+-+-")}


def _case(mode):
    if mode not in _CASES:
        tabs = _tables(mode == "stacking")
        _CASES[mode] = (tabs, [oracle_align(t, **MODES[mode]) for t in tabs])
    return _CASES[mode]


@pytest.mark.gpu
@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("lanes", [32, 64])
@pytest.mark.parametrize("budget", [-1, 0])
@pytest.mark.parametrize("device_index", ["0", "1"])
def test_mixed_chunks_match_oracle(engine, monkeypatch, mode, lanes, budget, device_index):
    tabs, ref = _case(mode)
    assert tabs[1].anchors is not None and max(tabs[-1].max_col) - min(tabs[-1].min_col) > 640
    monkeypatch.setenv("LCG_LANES", str(lanes))
    monkeypatch.setenv("LCG_DEVICE_INDEX", device_index)
    try:
        engine.set_rect_budget(budget)
        for chunk in (0, 4):
            engine.set_chunk_pairs(chunk)
            for _ in range(2):
                for k, (r, o) in enumerate(zip(engine.align_pairs(tabs, **MODES[mode]), ref)):
                    assert_same_result(r, o, f"pair {k}, chunks of {chunk}")
    finally:
        engine.set_rect_budget(-1)
        engine.set_chunk_pairs(0)


@pytest.mark.gpu
def test_wide_pair_in_a_pf_batch(engine, monkeypatch):
    """One pair past the limits: the FP32 batch goes to one warp per group; within
    1e-5 of FP64, as the FP32 passes are held to throughout."""
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_rna
    import numpy as np
    kw = dict(min_trace_probability=0.0, pf_precision=0)
    tabs = [prepare_pair(make_rna(a, a).to_pp(), make_rna(b, b).to_pp(), **kw) for a, b in [(60, 50), (24, 660), (33, 40)]]
    lz64 = engine.pf_forward(tabs, precision=64, min_am_prob=0.0, gap_gradients=False)
    r64 = engine.pf_backward()
    monkeypatch.setenv("LCG_LANES", "32")
    lz = engine.pf_forward(tabs, precision=32, min_am_prob=0.0, gap_gradients=False)
    for k, r in enumerate(engine.pf_backward()):
        assert abs(lz[k] - lz64[k]) <= 1e-5 * max(1.0, abs(lz64[k]))
        assert np.max(np.abs(r["am_prob"] - r64[k]["am_prob"]), initial=0.0) <= 1e-5
        assert np.max(np.abs(r["bm_prob"] - r64[k]["bm_prob"])) <= 1e-5
