"""LocARNA-P's top level by a block (pf_top_sweep, pf_top_back in
pf_kernels.cu) at widths around its 128 threads and rows of a few to some
hundred entries: log Z against the oracle, the gradients against central
differences of log Z (h = 1e-3: their error is below 1e-6 relative, 1e-4 is
allowed), with and without kept E and F."""
import math

import numpy as np
import pytest

from oracle_ffi import oracle_pf

H = 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("la,lb", [(8, 5), (30, 127), (31, 128), (25, 129), (20, 257), (130, 20), (90, 90)])
def test_top_level_widths(engine, la, lb):
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_rna
    a = make_rna(la, 40 + la)
    b = make_rna(lb, 60 + lb) if la != lb else make_homolog(a, 3)
    t = prepare_pair(a.to_pp(), b.to_pp(), min_trace_probability=0.0 if la != lb else 1e-5, pf_precision=0)
    z, _, _ = oracle_pf(t, probs=False)
    try:
        for budget in (-1, 0):
            engine.set_rect_budget(budget)
            lz = engine.pf_forward([t], precision=64, min_am_prob=0.0)[0]
            assert abs(lz - math.log(z)) <= 1e-10 * max(1.0, abs(lz))
            r = engine.pf_backward()[0]
            grads = [r["dlogz_dindel"], r["dlogz_dindel_opening"], r["dlogz_dstruct_weight"]] + list(r["dlogz_dbasematch"])
            for k, g in enumerate(grads):
                d = np.zeros(19)
                d[k] = H
                up = engine.pf_forward([t], precision=64, param_delta=d, min_am_prob=0.0)[0]
                down = engine.pf_forward([t], precision=64, param_delta=-d, min_am_prob=0.0)[0]
                fd = (up - down) / (2 * H)
                # (log Z itself is good to 1e-13 relative: 1e-10 in the quotient)
                assert abs(g - fd) <= 1e-4 * abs(fd) + 1e-9 * max(1.0, abs(lz)), (k, g, fd)
    finally:
        engine.set_rect_budget(-1)
