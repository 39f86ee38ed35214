"""The fill kernel for few items (sankoff_fill_kernel<AHEAD>: entries and values
read ahead) and the one for many, on single pairs on both sides of the line
between them, in every form the kernel takes, against the oracle. Whole numbers:
equal, no tolerance. Lane per group is off (LCG_LANES)."""
import pytest

from checks import assert_same_result
from oracle_ffi import oracle_align


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [dict(), dict(no_lonely_pairs=True), dict(stacking=1), dict(free_endgaps="++++"),
                                  dict(sequ_local=True), dict(profile=1)])
def test_fill_ahead_matches_oracle(engine, monkeypatch, mode):
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_profile, make_rna
    monkeypatch.setenv("LCG_LANES", "0")
    stack = mode.get("stacking", 0)
    kw = {k: v for k, v in mode.items() if k not in ("stacking", "profile")}
    prep = dict(stacking=1, exp_prob=0.01) if stack else {}
    for k, (la, lb) in enumerate([(4, 5), (33, 8), (60, 61), (40, 130), (150, 140), (230, 230)]):
        if mode.get("profile"):
            a, b = make_profile(la, 5 + k), make_profile(lb, 60 + k)
        else:
            a = make_rna(la, 300 + k)
            b = make_homolog(a, 7 + k) if k % 2 else make_rna(lb, 350 + k)
        kwp = dict(stacking=bool(stack)) if stack else {}
        t = prepare_pair(a.to_pp(**kwp), b.to_pp(**kwp), **prep)
        assert_same_result(engine.align_pairs([t], **kw)[0], oracle_align(t, **kw), f"{la} x {lb}")
