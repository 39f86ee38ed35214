"""Two engines in two threads, one with short pairs, one with long ones: a
kernel's limit of dynamic shared memory belongs to the process, so a call must
not lower it under a launch of the other thread. Results equal those of one
thread; the loops are long enough that setting and launch interleave."""
import threading

import numpy as np
import pytest


def _both(first, second, rounds):
    failed = []

    def work(fn):
        try:
            for _ in range(rounds):
                fn()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            failed.append(repr(e))

    th = [threading.Thread(target=work, args=(f,)) for f in (first, second)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not failed, failed


@pytest.mark.gpu
def test_envelopes_in_two_threads():
    from locarna_gb300.engine import Engine
    from locarna_gb300.prep import prepare_pairs
    from locarna_gb300.synth import make_rna
    runs = []
    for n, rounds in ((20, 400), (380, 400)):
        pairs = [(make_rna(n, 1).to_pp(), make_rna(n + 3, 2).to_pp())]
        eng = Engine(0)
        ref = prepare_pairs(eng, pairs)[0][0]

        def run(eng=eng, pairs=pairs, ref=ref):
            t = prepare_pairs(eng, pairs)[0][0]
            assert np.array_equal(t.min_col, ref.min_col) and np.array_equal(t.max_col, ref.max_col)
        runs.append(run)
    _both(*runs, 400)


def _wide(n, m, seed):
    """A pair without an envelope: the band spans all columns."""
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_rna
    return prepare_pair(make_rna(n, seed).to_pp(), make_rna(m, seed + 1).to_pp(), min_trace_probability=0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["fill", "lanes", "struct_local", "normalized", "pf64", "pf32", "pf_lanes"])
def test_engines_in_two_threads(monkeypatch, kind):
    from locarna_gb300.engine import Engine
    monkeypatch.setenv("LCG_LANES", {"lanes": "64", "pf_lanes": "32"}.get(kind, "0"))
    runs = []
    for n, m in ((12, 14), (40, 420)):
        t = _wide(n, m, n)
        eng = Engine(0)

        def run(eng=eng, t=t):
            if kind.startswith("pf"):
                lz = eng.pf_forward([t], precision=64 if kind == "pf64" else 32, min_am_prob=0.0,
                                    gap_gradients=kind != "pf_lanes")
                eng.pf_backward()
                return round(float(lz[0]), 2)
            kw = {"struct_local": dict(struct_local=True), "normalized": dict(sequ_local=True, normalized=50)}.get(kind, {})
            r = eng.align_pairs([t], **kw)[0]
            return r.score, r.edges
        ref = run()

        def check(run=run, ref=ref):
            assert run() == ref
        runs.append(check)
    _both(*runs, 300)
