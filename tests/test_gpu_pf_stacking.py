"""LocARNA-P of pairs that carry stacking tables: its recursions have no stacking
terms, so log Z and the probabilities are those of the same pairs without the
tables, whether the host or the device (LCG_DEVICE_INDEX) makes the index
structures. Both calls sum the same terms, in the order that atomics happen to
take: 1e-12 relative in FP64, 1e-6 in FP32."""
import copy

import numpy as np
import pytest


def _tables():
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_rna
    tabs = []
    for k, (la, lb) in enumerate([(16, 31), (64, 60), (120, 110)]):
        a = make_rna(la, 40 + k)
        b = make_homolog(a, 5) if k % 2 else make_rna(lb, 60 + k)
        tabs.append(prepare_pair(a.to_pp(stacking=True), b.to_pp(stacking=True), stacking=1, exp_prob=0.01,
                                 min_trace_probability=1e-5, pf_precision=0))
    return tabs


@pytest.mark.gpu
@pytest.mark.parametrize("precision,lanes", [(64, 0), (32, 0), (32, 32)])
@pytest.mark.parametrize("device_index", ["0", "1"])
def test_stacking_tables_are_ignored(engine, monkeypatch, precision, lanes, device_index):
    tabs = _tables()
    assert all(t.am_stack_score is not None and len(t.am_stack_score) for t in tabs)
    bare = [copy.copy(t) for t in tabs]
    for t in bare:
        t.am_stack_score = t.am_stackable = None
    monkeypatch.setenv("LCG_LANES", str(lanes))
    monkeypatch.setenv("LCG_DEVICE_INDEX", device_index)
    tol = 1e-12 if precision == 64 else 1e-6
    out = []
    for batch in (tabs, bare):
        lz = engine.pf_forward(batch, precision=precision, min_am_prob=0.0, gap_gradients=lanes == 0)
        out.append((lz, engine.pf_backward()))
    for k in range(len(tabs)):
        a, b = out[0][1][k], out[1][1][k]
        assert abs(out[0][0][k] - out[1][0][k]) <= tol * max(1.0, abs(out[1][0][k]))
        assert np.max(np.abs(a["am_prob"] - b["am_prob"]), initial=0.0) <= tol
        assert np.max(np.abs(a["bm_prob"] - b["bm_prob"])) <= tol
