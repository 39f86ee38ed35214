"""The envelope kernel at the sizes where its rows change shape: columns around
the warp's 32, one column or row, bands that cut a chunk, rows enough to be
rescaled, and lengths that differ by a lot; the tables equal the host path's."""
import pytest

from test_gpu_envelope import _same_tables


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [{}, {"max_diff": 7}, {"sequ_local": 1}, {"pf_precision": 0, "min_trace_probability": 1e-5}])
def test_envelope_sizes(engine, kw):
    from locarna_gb300.prep import prepare_pair, prepare_pairs
    from locarna_gb300.synth import make_homolog, make_rna
    pairs = []
    for k, (la, lb) in enumerate([(5, 5), (31, 32), (32, 31), (33, 33), (63, 64), (65, 62), (95, 97), (128, 127), (40, 161),
                                  (161, 40), (300, 290)]):
        a = make_rna(la, 60 + k)
        b = make_homolog(a, 5 + k) if abs(la - lb) < 2 or "sequ_local" in kw else make_rna(lb, 80 + k)
        pairs.append((a.to_pp(), b.to_pp()))
    got, nhost = prepare_pairs(engine, pairs, **kw)
    for k, ((a, b), t) in enumerate(zip(pairs, got)):
        _same_tables(t, prepare_pair(a, b, **kw), f"pair {k}")
    assert nhost <= 1
