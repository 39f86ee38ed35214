"""Envelopes of pairs whose match weights take most of FP64's range: long runs of
small weights, then a stem of weights up to 2^1000 (a very large structure weight),
at the ends and inside. The tables equal the host path's (long double), and the
envelopes are decided on the GPU: the weights fit FP64 as long as every row is
scaled on its own."""
import random

import pytest

from test_gpu_envelope import _same_tables


def _pp(n, at):
    from locarna_gb300.synth import RnaRecord
    rng = random.Random(5)
    seq = [rng.choice("ACGU") for _ in range(n)]
    pairs = {}
    for k in range(3):
        i, j = at + k, at + 12 - k
        seq[i - 1], seq[j - 1] = "G", "C"
        pairs[(i, j)] = 0.99
    return RnaRecord("r", "".join(seq), pairs).to_pp()


@pytest.mark.gpu
@pytest.mark.parametrize("struct_weight", [180000, 198500, 205000])
@pytest.mark.parametrize("kw", [{}, {"sequ_local": 1}, {"free_endgaps": "++++"}])
def test_envelope_range(engine, struct_weight, kw):
    from locarna_gb300.prep import prepare_pair, prepare_pairs
    pairs = [(_pp(n, at), _pp(n, at)) for n, at in [(110, 97), (150, 137), (200, 187), (200, 20), (240, 100)]]
    got, nhost = prepare_pairs(engine, pairs, struct_weight=struct_weight, **kw)
    for k, ((a, b), t) in enumerate(zip(pairs, got)):
        _same_tables(t, prepare_pair(a, b, struct_weight=struct_weight, **kw), f"pair {k}")
    assert nhost == 0
