"""LocARNA-P in FP32 lane per group (pf_lane_kernels.cu), forced on for every
size (LCG_LANES), against the FP64 passes: log Z within 1e-5 relative and
probabilities within 1e-5 absolute, the bounds the FP32 passes are held to
throughout. Sizes at the edges of the 8-column blocks and 4-row quads, items of a
few groups to many, uses and seeds in one quad (homologs), dense weights
(profiles), exact and truncated base-match sums, M kept and swept again."""
import numpy as np
import pytest

TOL = 1e-5
SIZES = [(9, 12), (15, 16), (17, 31), (33, 24), (40, 41), (64, 60), (96, 71), (50, 120), (130, 140)]


def _tables():
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_profile, make_rna
    kw = dict(min_trace_probability=1e-5, pf_precision=0)
    tabs = []
    for k, (la, lb) in enumerate(SIZES):
        a = make_rna(la, 900 + k)
        b = make_homolog(a, 7 + k) if k % 2 else make_rna(lb, 950 + k)
        tabs.append(prepare_pair(a.to_pp(), b.to_pp(), **kw))
    tabs.append(prepare_pair(make_profile(60, 5).to_pp(), make_profile(52, 6).to_pp(), **kw))
    return tabs


@pytest.mark.gpu
@pytest.mark.parametrize("min_am_prob", [0.0, 0.001])
@pytest.mark.parametrize("budget", [-1, 0])
@pytest.mark.parametrize("single", [False, True])
def test_pf_lanes_match_fp64(engine, monkeypatch, min_am_prob, budget, single):
    tabs = _tables()
    lz64 = engine.pf_forward(tabs, precision=64, min_am_prob=min_am_prob, gap_gradients=False)
    r64 = engine.pf_backward()
    monkeypatch.setenv("LCG_LANES", "32")
    try:
        engine.set_rect_budget(budget)
        for batch in ([[k] for k in range(len(tabs))] if single else [list(range(len(tabs)))]):
            lz = engine.pf_forward([tabs[k] for k in batch], precision=32, min_am_prob=min_am_prob, gap_gradients=False)
            for i, (k, r) in enumerate(zip(batch, engine.pf_backward())):
                assert abs(lz[i] - lz64[k]) <= TOL * max(1.0, abs(lz64[k]))
                assert np.max(np.abs(r["am_prob"] - r64[k]["am_prob"]), initial=0.0) <= TOL
                assert np.max(np.abs(r["bm_prob"] - r64[k]["bm_prob"])) <= TOL
                assert abs(r["dlogz_dstruct_weight"] - r64[k]["dlogz_dstruct_weight"]) <= TOL * max(
                    1.0, abs(r64[k]["dlogz_dstruct_weight"]))
    finally:
        engine.set_rect_budget(-1)
