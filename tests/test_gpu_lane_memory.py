"""Device memory of a batch filled lane per group (sankoff_lane_kernels.cu) under a
caller's budget: with lcg_engine_set_rect_budget(0) it takes no more than the same
batch filled by one warp per group, but for the tables that the lane items add (64
MB is ample for 45 pairs). Results are equal in every case."""
import pytest


@pytest.mark.gpu
def test_budget_bounds_the_lane_slots(monkeypatch):
    torch = pytest.importorskip("torch")
    from locarna_gb300.engine import Engine
    from locarna_gb300.prep import prepare_pairs
    from locarna_gb300.synth import make_rna
    pp = [make_rna(n, n).to_pp() for n in range(290, 300)]
    eng = Engine(0)
    tabs, _ = prepare_pairs(eng, [(pp[a], pp[b]) for a in range(10) for b in range(a + 1, 10)])
    ref = [(r.score, r.edges) for r in eng.align_pairs(tabs)]
    taken = {}
    for lanes in ("0", "64", "32"):
        monkeypatch.setenv("LCG_LANES", lanes)
        eng = Engine(0)
        eng.set_rect_budget(0)
        free = torch.cuda.mem_get_info()[0]
        assert [(r.score, r.edges) for r in eng.align_pairs(tabs)] == ref
        taken[lanes] = free - torch.cuda.mem_get_info()[0]
        eng.set_rect_budget(-1)
        assert [(r.score, r.edges) for r in eng.align_pairs(tabs)] == ref
        del eng
    assert max(taken["32"], taken["64"]) <= taken["0"] + (64 << 20), taken
