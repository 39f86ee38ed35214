"""Calls with less device memory than they ask for at first. The test builds a
variant of the library (its own folder; only the host code is compiled again)
whose allocations above $LCG_TEST_ALLOC_BYTES are refused (LCG_TEST_ALLOC), so
that no GPU is filled. A child process runs each call without and with the
limit, twice with it, and compares."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = textwrap.dedent("""
    import os, sys
    sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
    import numpy as np
    import locarna_gb300.engine as E
    E.load_library({lib!r})
    from locarna_gb300.engine import Engine
    from locarna_gb300.prep import prepare_pairs
    from locarna_gb300.synth import make_rna
    def limit(nbytes):
        os.environ.pop("LCG_TEST_ALLOC_BYTES", None)
        if nbytes:
            os.environ["LCG_TEST_ALLOC_BYTES"] = str(nbytes)
    pp = [make_rna(n, 30 + n).to_pp() for n in (60, 85, 110, 140, 200)]
    pairs = [(pp[a], pp[b]) for a in range(5) for b in range(a + 1, 5)]
""")


@pytest.fixture(scope="module")
def child():
    from locarna_gb300.build import OUT, build_engine
    build_engine()
    out = os.path.join(OUT, "alloc_limit_test")
    os.makedirs(out, exist_ok=True)
    for f in os.listdir(OUT):
        if f.endswith(".o") and f not in ("engine.cu.o", "engine_pf.cu.o", "envelope.cu.o"):
            shutil.copy2(os.path.join(OUT, f), out)
    lib = build_engine(out=out, defs=["-DLCG_TEST_ALLOC"])
    head = HEAD.format(root=ROOT, tests=os.path.join(ROOT, "tests"), lib=lib)

    def run(code):
        r = subprocess.run([sys.executable, "-c", head + textwrap.dedent(code)], capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
        return r.stderr  # one line "refused <bytes>" per refused allocation
    return run


# pairs of 0.3 to 1.6 MB, 7.7 MB together; under 1 MiB the two largest go to the
# host and the others in waves of one to three
@pytest.mark.gpu
def test_envelopes_in_smaller_waves(child):
    child("""
        ref, nhost = prepare_pairs(Engine(0), pairs)
        assert nhost == 0
        eng = Engine(0)
        for nbytes, hosts in ((1 << 20, 2), (1 << 20, 2), (4 << 20, 0)):
            limit(nbytes)
            got, nhost = prepare_pairs(eng, pairs)
            assert nhost == hosts, nhost
            for t, r in zip(got, ref):
                for f in ("min_col", "max_col", "am_arcs", "am_score"):
                    assert np.array_equal(getattr(t, f), getattr(r, f)), f
                assert t.envelope_ok == r.envelope_ok
        print("ok")
    """)


# ten pairs with whole bands: the items' storage (1.8 GB) and the slots of all warps
# (6.0 GB) are refused at every limit; one warp per group takes 0.5 GB of scratch, so
# the batch goes there at 900 MB and to a few blocks of lanes below. The second call
# makes no attempt that has failed before, setting the budget forgets them.
@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [32, 64])
@pytest.mark.parametrize("megabytes", [900, 300, 150])
def test_lane_fill_with_less_memory(child, lanes, megabytes):
    err = child(f"""
        os.environ["LCG_LANES"] = "{lanes}"
        tabs, _ = prepare_pairs(Engine(0), pairs, min_trace_probability=0.0)
        ref = [(r.score, r.edges) for r in Engine(0).align_pairs(tabs)]
        eng = Engine(0)
        limit({megabytes} << 20)
        for k in range(2):
            assert [(r.score, r.edges) for r in eng.align_pairs(tabs)] == ref
            print("call", k, file=sys.stderr, flush=True)
        eng.set_rect_budget(-1)
        assert [(r.score, r.edges) for r in eng.align_pairs(tabs)] == ref
        print("ok")
    """)
    first, second, third = err.split("call")
    assert "refused" in first and "refused" not in second and "refused" in third, err


# (one warp per group takes 2.2 GB here: 3000 MB goes there)
@pytest.mark.gpu
@pytest.mark.parametrize("megabytes", [3000, 900, 300, 150])
def test_pf_lanes_with_less_memory(child, megabytes):
    err = child(f"""
        os.environ["LCG_LANES"] = "32"
        kw = dict(precision=32, min_am_prob=0.0, gap_gradients=False)
        tabs, _ = prepare_pairs(Engine(0), pairs, min_trace_probability=0.0, pf_precision=0)
        ref = Engine(0)
        lz = ref.pf_forward(tabs, **kw)
        probs = ref.pf_backward()
        eng = Engine(0)
        limit({megabytes} << 20)
        for k in range(2):
            got = eng.pf_forward(tabs, **kw)
            assert np.max(np.abs(np.array(got) - np.array(lz)) / np.maximum(1.0, np.abs(lz))) <= 1e-5
            for r, p in zip(eng.pf_backward(), probs):
                assert np.max(np.abs(r["am_prob"] - p["am_prob"]), initial=0.0) <= 1e-5
                assert np.max(np.abs(r["bm_prob"] - p["bm_prob"])) <= 1e-5
            print("call", k, file=sys.stderr, flush=True)
        print("ok")
    """)
    first, second, _ = err.split("call")
    assert "refused" in first and "refused" not in second, err


# 190 pairs of 55-64 nt in chunks of 40: the envelopes of the pairs behind the first
# chunk (31 MB at once) are refused where they are enqueued for later, and done in
# waves; a chunk of the alignment takes less
@pytest.mark.gpu
def test_later_envelopes_in_waves(child):
    err = child("""
        lens = [55 + k % 10 for k in range(20)]
        rnas = [make_rna(n, 200 + k).to_pp() for k, n in enumerate(lens)]
        ids = [(a, b) for a in range(20) for b in range(a + 1, 20)]
        out = []
        for nbytes in (0, 30 << 20):
            eng = Engine(0)
            eng.set_chunk_pairs(40)
            os.environ["LCG_LANES"] = "32"
            call = eng.prepare_pp_call([(rnas[a], rnas[b]) for a, b in ids], [(lens[a], lens[b]) for a, b in ids])
            limit(nbytes)
            for _ in range(2):
                assert eng.run_pp_call(call) == 0
                out.append([(r.score, r.edges) for r in Engine.decode_pp_call(call)])
                print("call", file=sys.stderr, flush=True)
        assert all(o == out[0] for o in out)
        print("ok")
    """)
    assert "refused 3" in err.split("call")[2] and "refused" not in err.split("call")[3], err
