"""Index structures made on the device (index_kernels.cu) against those of the
host (LCG_DEVICE_INDEX = 1 / 0): equal results on the reference's golden cases
and on pairs of a few nt, and arcs or arc matches in another order than
ArcMatches', which the host path takes."""
import numpy as np
import pytest

from checks import assert_kbest_matches_golden, assert_matches_golden, assert_same_result
from golden_io import Golden, sankoff_golden_names
from locarna_gb300.abi import PairTables
from oracle_ffi import oracle_align


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", ["0", "32"])
@pytest.mark.parametrize("name", [n for n in sankoff_golden_names() if not n.startswith("c400")])
def test_device_index_matches_reference(engine, monkeypatch, name, lanes):
    monkeypatch.setenv("LCG_DEVICE_INDEX", "1")
    monkeypatch.setenv("LCG_LANES", lanes)
    g = Golden(name)
    kw = g.align_kwargs()
    if g.kbest:
        assert_kbest_matches_golden(g, engine.align_kbest([g.tables], *g.kbest, **kw)[0])
    else:
        assert_matches_golden(g, engine.align_pairs([g.tables], **kw)[0])


def _tables(stack):
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_rna
    out = []
    for k, (la, lb) in enumerate([(5, 5), (8, 9), (12, 31), (32, 33), (47, 40), (90, 64)]):
        a = make_rna(la, 700 + k)
        b = make_homolog(a, 3 + k) if k % 2 else make_rna(lb, 750 + k)
        kw = dict(stacking=1, exp_prob=0.01) if stack else {}
        out.append(prepare_pair(a.to_pp(stacking=stack), b.to_pp(stacking=stack), **kw))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("stack", [False, True])
@pytest.mark.parametrize("lanes", ["0", "64"])
def test_device_index_of_short_pairs(engine, monkeypatch, lanes, stack):
    monkeypatch.setenv("LCG_DEVICE_INDEX", "1")
    monkeypatch.setenv("LCG_LANES", lanes)
    tabs = _tables(stack)
    for k, (r, t) in enumerate(zip(engine.align_pairs(tabs), tabs)):
        assert_same_result(r, oracle_align(t), f"pair {k}")


def _renumbered(t, order_a, am_order):
    """The same pair with the arcs of A and the arc matches in another order."""
    arcs = t.arcs_a.reshape(-1, 2)[order_a]
    back = np.argsort(order_a)
    am = t.am_arcs.reshape(-1, 2).copy()
    am[:, 0] = back[am[:, 0]]
    return PairTables(t.len_a, t.len_b, t.sigma, t.gap_a, t.gap_b, t.indel_opening, t.exclusion, arcs, t.arcs_b,
                      am[am_order], t.am_score[am_order], t.min_col, t.max_col)


@pytest.mark.gpu
def test_other_orders_take_the_host_path(engine, monkeypatch):
    monkeypatch.setenv("LCG_DEVICE_INDEX", "1")
    t = _tables(False)[-1]
    want = engine.align_pairs([t])[0]
    na, nm = t.num_arcs_a, t.num_arcmatches
    rng = np.random.RandomState(4)
    same_a, same_m = np.arange(na), np.arange(nm)
    for order_a, order_m in [(same_a[::-1], same_m), (same_a, rng.permutation(nm)), (rng.permutation(na), same_m[::-1])]:
        u = _renumbered(t, order_a, order_m)
        got = engine.align_pairs([u])[0]
        assert (got.score, got.max_ij) == (want.score, want.max_ij)
        assert_same_result(got, oracle_align(u))
