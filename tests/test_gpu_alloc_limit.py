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
