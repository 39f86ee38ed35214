"""LocARNA-P with the index structures, the arc matches' weights and the
probabilities made on the device (LCG_DEVICE_INDEX): results as with the host's
index. Both sum the same terms, in the order that shared-memory and global
atomics happen to take: 1e-12 relative in FP64, 1e-6 in FP32, the bounds the
other comparisons of this kind use."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision,lanes", [(64, 0), (32, 0), (32, 32)])
@pytest.mark.parametrize("min_am_prob", [0.0, 0.001])
def test_pf_device_index(engine, monkeypatch, precision, lanes, min_am_prob):
    from locarna_gb300.prep import prepare_pair
    from locarna_gb300.synth import make_homolog, make_rna
    tabs = []
    for k, (la, lb) in enumerate([(5, 6), (16, 31), (64, 60), (33, 100), (120, 120)]):
        a = make_rna(la, 70 + k)
        b = make_homolog(a, 3) if la == lb else make_rna(lb, 80 + k)
        tabs.append(prepare_pair(a.to_pp(), b.to_pp(), min_trace_probability=1e-5, pf_precision=0))
    delta = np.zeros(19)
    delta[2] = 0.25  # the structure weight's offset goes through the arc matches' derivatives
    monkeypatch.setenv("LCG_LANES", str(lanes))
    tol = 1e-12 if precision == 64 else 1e-6
    out = []
    for dev in ("0", "1"):
        monkeypatch.setenv("LCG_DEVICE_INDEX", dev)
        lz = engine.pf_forward(tabs, precision=precision, min_am_prob=min_am_prob, param_delta=delta,
                               gap_gradients=lanes == 0)
        out.append((lz, engine.pf_backward()))
    for k in range(len(tabs)):
        a, b = out[0][1][k], out[1][1][k]
        assert abs(out[0][0][k] - out[1][0][k]) <= tol * max(1.0, abs(out[0][0][k]))
        assert np.max(np.abs(a["am_prob"] - b["am_prob"]), initial=0.0) <= tol
        assert np.max(np.abs(a["bm_prob"] - b["bm_prob"])) <= tol
        assert abs(a["dlogz_dstruct_weight"] - b["dlogz_dstruct_weight"]) <= tol * max(1.0, abs(a["dlogz_dstruct_weight"]))
        assert np.max(np.abs(a["dlogz_dbasematch"] - b["dlogz_dbasematch"])) <= tol * max(
            1.0, np.max(np.abs(a["dlogz_dbasematch"])))
