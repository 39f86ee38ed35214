"""The lane-per-group fill (sankoff_lane_kernels.cu) on a GPU, forced on for
pairs and batches of every size (LCG_LANES: groups per item), against the
reference's golden results and the oracle. Scores, tracebacks and end cells
are whole numbers: equal, no tolerance."""
import pytest

from checks import assert_kbest_matches_golden, assert_matches_golden, assert_same_result
from golden_io import Golden, sankoff_golden_names
from oracle_ffi import oracle_align

NAMES = sankoff_golden_names()


@pytest.fixture(params=[32, 64])
def lanes(request, monkeypatch):
    monkeypatch.setenv("LCG_LANES", str(request.param))
    return request.param


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_lanes_match_reference(engine, lanes, name):
    g = Golden(name)
    if g.struct_local:
        pytest.skip("structure-local alignment does not take this fill")
    kw = g.align_kwargs()
    if g.kbest:
        k, threshold = g.kbest
        assert_kbest_matches_golden(g, engine.align_kbest([g.tables], k, threshold, **kw)[0])
        return
    for budget in (-1, 0):  # traceback on the items' kept storage, and recomputing
        try:
            engine.set_rect_budget(budget)
            assert_matches_golden(g, engine.align_pairs([g.tables], **kw)[0])
        finally:
            engine.set_rect_budget(-1)


# one call over pairs of a few to some hundred nt (edges of the 8-column
# blocks and 4-row quads, one or many items), in the modes that change the D
# writes and the top level
@pytest.mark.gpu
@pytest.mark.parametrize("mode", [dict(), dict(no_lonely_pairs=True), dict(stacking=1),
                                  dict(no_lonely_pairs=True, stacking=1), dict(free_endgaps="++++"),
                                  dict(sequ_local=True), dict(sequ_local=True, normalized=50)])
def test_lane_batches_match_oracle(engine, lanes, mode):
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_profile, make_rna
    stack = mode.get("stacking", 0)
    kw = {k: v for k, v in mode.items() if k != "stacking"}
    prep = dict(stacking=1, exp_prob=0.01) if stack else {}
    tabs = []
    for k, (la, lb) in enumerate([(9, 12), (15, 16), (17, 31), (33, 24), (40, 41), (64, 60), (96, 71), (50, 120)]):
        a = make_rna(la, 900 + k)
        b = make_homolog(a, 7 + k) if k % 2 else make_rna(lb, 950 + k)
        tabs.append(prepare_pair(a.to_pp(stacking=bool(stack)), b.to_pp(stacking=bool(stack)), **prep))
    if not stack:
        tabs.append(prepare_pair(make_profile(60, 5).to_pp(), make_profile(52, 6).to_pp()))  # dense scores
    for k, (r, t) in enumerate(zip(engine.align_pairs(tabs, **kw), tabs)):
        assert_same_result(r, oracle_align(t, **kw), f"pair {k}")
