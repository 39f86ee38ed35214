"""The work a user of this library has it do, as cases that can be timed and compared.

A case names a kind of call (`kind`) with its sizes and options:

  align    lcg_align_pairs on prepared tables (`Engine.run_call`): the alignment of the pairs of one batch
  pp       lcg_align_pp_pairs (`Engine.run_pp_call`): PP texts in, alignments out
  pf       lcg_pf_forward + lcg_pf_backward (`Engine.pf_forward` / `pf_backward`): LocARNA-P

A case with `rnas` = 0 is one pair of `len_lo` x `len_hi` nt; otherwise all pairs of `rnas` RNAs whose lengths are spread
over [len_lo, len_hi] (uneven by construction, the same for every seed). The bases, the planted stems and the base-pair
probabilities come from the seed (locarna_gb300/synth.py).

`run` returns whole numbers for alignments (scores, end cells, edges, traced arc matches) and floating-point values for
LocARNA-P. LocARNA-P computed in FP32 is handed on as float32, the precision it has.
"""
import ctypes
import math

import numpy as np

from locarna_gb300.abi import lcg_align_result, make_opts
from locarna_gb300.engine import Engine
from locarna_gb300.prep import prepare_pairs
from locarna_gb300.synth import make_homolog, make_profile, make_rna

_ENGINE = None


def _engine():
    """The one engine of the process, as a program keeps it."""
    global _ENGINE
    if _ENGINE is None:
        _ENGINE = Engine(0)
    return _ENGINE


# ---------------------------------------------------------------- the cases


def _align(name, len_lo, len_hi, rnas=0, mode="global", data="rna"):
    return dict(name=name, kind="align", rnas=rnas, len_lo=len_lo, len_hi=len_hi, mode=mode, data=data)


def listed():
    return [
        # the smallest call: one short pair (an interactive or per-pair caller); latency
        _align("pair_60", 60, 57),
        # one ordinary pair, default scoring
        _align("pair_150", 150, 150),
        # one long pair, global and structure-local: the per-pair sizes of the long-RNA workload
        _align("pair_400", 400, 400),
        _align("pair_400_struct_local", 400, 400, mode="struct_local"),
        # all pairs of a family of uneven RNAs (the pairwise stage of a multiple alignment), tables at hand
        _align("allpairs_24", 60, 400, rnas=24),
        # the same stage from PP texts to alignments, the largest call
        dict(name="pp_allpairs_32", kind="pp", rnas=32, len_lo=60, len_hi=400, mode="global", data="rna"),
        # progressive alignment: profiles against profiles (averaged scores: no class table)
        _align("profiles_8", 80, 300, rnas=8, data="profile"),
        # related RNAs with stacking probabilities
        _align("stacking_10", 100, 300, rnas=10, mode="stacking", data="homolog"),
        # local alignment normalized by length (Dinkelbach iterations)
        _align("normalized_12", 60, 300, rnas=12, mode="normalized"),
        # LocARNA-P: one pair in FP64 with exact marginals and every gradient (forward and backward)
        dict(name="pf64_pair_200", kind="pf", rnas=0, len_lo=200, len_hi=200, precision=64, min_am_prob=0.0, grads=True),
        # LocARNA-P over a family in FP32: the probabilities for probabilistic consistency
        dict(name="pf32_allpairs_7", kind="pf", rnas=7, len_lo=80, len_hi=500, precision=32, min_am_prob=0.0,
             grads=False),
        # LocARNA-P over a family as the command line runs it: FP64, truncated base-match probabilities
        dict(name="pf64_allpairs_5", kind="pf", rnas=5, len_lo=80, len_hi=240, precision=64, min_am_prob=0.001,
             grads=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "batch", "batch", "profile", "pp", "pf_pair", "pf_batch"])
    if kind == "pair":
        c = _align("", _log_int(rng, 40, 400), _log_int(rng, 40, 400),
                   mode=rng.choice(["global", "global", "struct_local", "stacking", "nolp", "free_endgaps"]))
    elif kind == "batch":
        lo = _log_int(rng, 40, 200)
        c = _align("", lo, min(400, lo + rng.randint(10, 250)), rnas=_log_int(rng, 3, 24),
                   mode=rng.choice(["global", "global", "stacking", "nolp", "local", "normalized", "penalized"]),
                   data=rng.choice(["rna", "homolog"]))
    elif kind == "profile":
        lo = _log_int(rng, 50, 180)
        c = _align("", lo, lo + rng.randint(5, 120), rnas=rng.randint(2, 8), data="profile")
    elif kind == "pp":
        lo = _log_int(rng, 40, 150)
        c = dict(kind="pp", rnas=_log_int(rng, 3, 30), len_lo=lo, len_hi=min(400, lo + rng.randint(10, 250)),
                 mode=rng.choice(["global", "local", "nolp"]), data="rna")
    elif kind == "pf_pair":
        c = dict(kind="pf", rnas=0, len_lo=_log_int(rng, 60, 300), len_hi=_log_int(rng, 60, 300),
                 precision=rng.choice([32, 64]), min_am_prob=rng.choice([0.0, 0.001]), grads=rng.choice([True, False]))
    else:
        lo = _log_int(rng, 60, 160)
        c = dict(kind="pf", rnas=rng.randint(3, 6), len_lo=lo, len_hi=lo + rng.randint(10, 200),
                 precision=rng.choice([32, 64]), min_am_prob=rng.choice([0.0, 0.001]), grads=False)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- inputs


def _lengths(case):
    if not case["rnas"]:
        return [case["len_lo"], case["len_hi"]]
    span = case["len_hi"] - case["len_lo"]
    return [case["len_lo"] + int((0.382 + 0.618034 * k) % 1.0 * (span + 1)) for k in range(case["rnas"])]


def _pairs(count):
    return [(a, b) for a in range(count) for b in range(a + 1, count)]


def _texts(case, seed):
    """One PP text per RNA (or profile) of the case."""
    stack = case.get("mode") == "stacking"
    out = []
    for k, n in enumerate(_lengths(case)):
        s = 100003 * (int(seed) + 1) + k
        if case.get("data") == "profile":
            out.append(make_profile(n, s, nrows=2 + k % 3).to_pp())
            continue
        rec = make_rna(n, s)
        if case.get("data") == "homolog" and k % 2:
            rec = make_homolog(make_rna(n, 100003 * (int(seed) + 1) + k - 1), s)
        out.append(rec.to_pp(stacking=stack))
    return out


def _options(mode):
    """(preparation options, alignment options) of an alignment mode; every mode aligns the default tables."""
    return {
        "global": (dict(), dict()),
        "struct_local": (dict(), dict(struct_local=True)),
        "stacking": (dict(stacking=1, exp_prob=0.01), dict()),
        "nolp": (dict(), dict(no_lonely_pairs=True)),
        "free_endgaps": (dict(), dict(free_endgaps="++++")),
        "local": (dict(), dict(sequ_local=True)),
        "normalized": (dict(), dict(sequ_local=True, normalized=100)),
        "penalized": (dict(), dict(sequ_local=True, penalized=50)),
    }[mode]


class _Results:
    """Caller-owned result buffers of a batch: one array for all edges and one for all traced arc matches."""

    def __init__(self, lens):
        n = len(lens)
        self.c = (lcg_align_result * n)()
        e_at = np.cumsum([0] + [2 * (a + b) + 2 for a, b in lens])
        t_at = np.cumsum([0] + [min(a, b) + 1 for a, b in lens])
        self.edges = np.zeros(int(e_at[-1]), np.int32)
        self.traced = np.zeros(int(t_at[-1]), np.int32)
        p32 = ctypes.POINTER(ctypes.c_int32)
        for k in range(n):
            self.c[k].edges = ctypes.cast(self.edges.ctypes.data + 4 * int(e_at[k]), p32)
            self.c[k].traced_am = ctypes.cast(self.traced.ctypes.data + 4 * int(t_at[k]), p32)
        words = ctypes.sizeof(lcg_align_result) // 8
        self.words = np.frombuffer(self.c, dtype=np.int64).reshape(n, words)

    def outputs(self):
        # per pair the score, the end cells and the edge and arc-match counts (the struct without its two pointers)
        return {"results": self.words[:, :4], "edges": self.edges, "traced_am": self.traced}


def prepare(case, seed):
    eng = _engine()
    pp = _texts(case, seed)
    ids = _pairs(len(pp))
    texts = [(pp[a], pp[b]) for a, b in ids]
    lens = _lengths(case)
    if case["kind"] == "pf":
        tables, _ = prepare_pairs(eng, texts, min_trace_probability=1e-5, pf_precision=0)
        return dict(kind="pf", tables=tables, precision=case["precision"], min_am_prob=case["min_am_prob"],
                    grads=case["grads"])
    popts, aopts = _options(case["mode"])
    buf = _Results([(lens[a], lens[b]) for a, b in ids])
    if case["kind"] == "pp":
        call = list(eng.prepare_pp_call(texts, [(lens[a], lens[b]) for a, b in ids], **aopts))
        if popts:
            from locarna_gb300.prep import prep_options
            call[3] = prep_options(**popts)
        call[5] = buf.c
        return dict(kind="pp", call=tuple(call), buf=buf)
    tables, _ = prepare_pairs(eng, texts, **popts)
    arr = (type(tables[0].to_c()) * len(tables))(*[t.to_c() for t in tables])
    return dict(kind="align", call=(arr, len(tables), make_opts(**aopts), buf.c, None, tables), buf=buf)


def _padded(am_prob, t, kind):
    """The arc-match probabilities of a pair, with zeros behind them up to a length that its sequence lengths alone give
    (how many arc matches there are depends on the seed)."""
    out = np.zeros(200 + 4 * t.len_a * t.len_b, kind)
    out[:len(am_prob)] = am_prob
    return out


def run(state):
    eng = _engine()
    if state["kind"] == "align":
        eng.run_call(state["call"])
        return state["buf"].outputs()
    if state["kind"] == "pp":
        eng.run_pp_call(state["call"])
        return state["buf"].outputs()
    single = state["precision"] == 32
    eng.pf_forward(state["tables"], precision=state["precision"], min_am_prob=state["min_am_prob"],
                   gap_gradients=state["grads"])
    kind = np.float32 if single else np.float64
    out = []
    for t, r in zip(state["tables"], eng.pf_backward()):
        o = {"log_z": np.array([r["log_z"]], kind), "am_prob": _padded(r["am_prob"], t, kind),
             "bm_prob": r["bm_prob"].astype(kind, copy=False)}
        if state["grads"]:
            o["grads"] = np.array([r["dlogz_dindel"], r["dlogz_dindel_opening"], r["dlogz_dstruct_weight"],
                                   *r["dlogz_dbasematch"]], kind)
        out.append(o)
    return out


# ---------------------------------------------------------------- work


def work(case):
    """Estimates from the sizes. The matrix cells of all left-end groups of a pair grow like the square of the matrix
    (0.0085 (n m)^2 within a few tens of per cent for these RNAs), with about one arc-match term per cell: 12 integer
    operations a cell for an alignment (8 times that in the eight-state structure-local mode), 14 a cell forward and 40
    backward for LocARNA-P. Lonely pairs excluded: a fiftieth of the cells. Inputs and outputs, each once: the
    base-match table, the arc matches (12 B each, about 1.4e-5 (n m)^1.9 of them) and the results (LocARNA-P: a
    probability per base match and per arc match)."""
    lens = _lengths(case)
    pf = case["kind"] == "pf"
    cells = nbytes = 0.0
    for a, b in _pairs(len(lens)):
        nm = float(lens[a]) * lens[b]
        cells += 0.0085 * nm * nm
        ams = 1.4e-5 * nm ** 1.9
        nbytes += 4 * nm + 12 * ams + 16 * (lens[a] + lens[b]) + (8 * (nm + ams) if pf else 0)
    if case.get("mode") == "nolp":
        cells /= 50
    per_cell = 54 if pf else 96 if case["mode"] == "struct_local" else 12
    if pf and case["min_am_prob"] > 0:
        per_cell += 20
    return {"bytes": nbytes, "flops": cells * per_cell}


# ---------------------------------------------------------------- LocARNA-P in 64 bits


def _pf_exact(t, min_am_prob, grads, temp=300.0):
    """LocARNA-P of one pair in plain numpy: the sum over alignments with weights exp(score / T), inside by rows with all
    left-end groups as one vector per cell, and its adjoint by the same sweep backwards.

    A group is a left-end pair (al, bl); group 0 is the top level (0, 0). Per cell (i, j) the vectors cover the groups
    with al < i, a prefix in ascending order of al."""
    n, m = t.len_a, t.len_b
    lo, hi = t.min_col.astype(int), t.max_col.astype(int)
    arc_a, arc_b = t.arcs_a.reshape(-1, 2), t.arcs_b.reshape(-1, 2)
    am = t.am_arcs.reshape(-1, 2)
    al, ar = (arc_a[am[:, 0], c].astype(int) for c in (0, 1)) if len(am) else (np.zeros(0, int),) * 2
    bl, br = (arc_b[am[:, 1], c].astype(int) for c in (0, 1)) if len(am) else (np.zeros(0, int),) * 2
    bm = np.exp(t.sigma.reshape(n + 1, m + 1) / temp)
    g_a, g_b = np.exp(t.gap_a / temp), np.exp(t.gap_b / temp)
    op, w = math.exp(t.indel_opening / temp), np.exp(t.am_score / temp)

    def inside(i, j):
        return (lo[i] <= j) & (j <= hi[i])

    use = inside(ar, br) & inside(al, bl) & inside(al - 1, bl - 1) & inside(ar - 1, br - 1)
    keys = sorted({(0, 0)} | set(zip(al[use].tolist(), bl[use].tolist())))
    number = {k: g for g, k in enumerate(keys)}
    ga, gb = np.array([k[0] for k in keys]), np.array([k[1] for k in keys])
    started = [int(np.searchsorted(ga, i, "left")) for i in range(n + 2)]  # groups with al < i
    ends_at, makes = {}, {}
    for k in np.nonzero(use)[0].tolist():
        ends_at.setdefault((ar[k], br[k]), []).append(k)
        makes.setdefault((ar[k] - 1, br[k] - 1), []).append(k)
    group_of = np.array([number.get((a, b), -1) for a, b in zip(al.tolist(), bl.tolist())], int)
    d = np.zeros(len(am))
    mat, ext, ins = {}, {}, {}  # M, E and F per cell, over the groups that have started
    for i in range(n + 1):
        p, p1 = started[i], started[i + 1]
        q_left = f_left = None
        for j in range(lo[i], hi[i] + 1):
            x, e = np.zeros(p1), np.zeros(p1)
            if i and j and (i - 1, j - 1) in mat:
                x[:p] = mat[i - 1, j - 1] * bm[i, j]
            if i and (i - 1, j) in mat:
                e[:p] = g_a[i] * (ext[i - 1, j] + op * (mat[i - 1, j] - ext[i - 1, j]))
            for k in ends_at.get((i, j), ()):
                c = mat[al[k] - 1, bl[k] - 1]
                x[:len(c)] += c * d[k]
            x[p:][gb[p:p1] == j] = 1.0  # M(al, bl) of the groups that start in this row
            f = g_b[j] * (f_left + op * q_left) if q_left is not None else np.zeros(p1)
            mat[i, j], ext[i, j], ins[i, j] = x + e + f, e, f
            q_left, f_left = x + e, f
            for k in makes.get((i, j), ()):
                d[k] = mat[i, j][group_of[k]] * w[k]
    z = mat[n, m][0]

    def back(seeds, nested):
        """Sum of X_bar M bm per cell, d Z / d D and the expected gap positions and openings (times Z) for the adjoint
        seeded at M(n, m) of the top level and, if `nested`, through every arc match; else at the given ones alone."""
        d_bar, uses, n_ext, n_open = np.zeros(len(am)), np.zeros((n + 1, m + 1)), 0.0, 0.0
        bar = {(n, m): np.eye(1, started[n + 1])[0]}
        e_down = {}  # E_bar of row i + 1 by column
        for i in range(n, -1, -1):
            p, p1 = started[i], started[i + 1]
            e_here, f_bar, f_right_col = {}, None, None
            for j in range(hi[i], lo[i] - 1, -1):
                b = bar.pop((i, j), None)
                b = np.zeros(p1) if b is None else b
                for k in makes.get((i, j), ()):
                    if nested:
                        b[group_of[k]] += d_bar[k] * w[k]
                    elif k in seeds:
                        b[group_of[k]] += seeds[k] * w[k]
                # M = X + E + F; N = X + F feeds E(i+1, j), Q = X + E feeds F(i, j+1)
                n_bar, e_next = np.zeros(p1), np.zeros(p1)
                if j in e_down:
                    v = e_down[j][:p1]
                    n_bar, e_next = v * g_a[i + 1] * op, v * g_a[i + 1]
                q_bar, f_next = np.zeros(p1), np.zeros(p1)
                if f_bar is not None:
                    q_bar, f_next = f_bar * g_b[j + 1] * op, f_bar * g_b[j + 1]
                x_bar, e_bar, f_now = b + n_bar + q_bar, b + q_bar + e_next, b + n_bar + f_next
                n_ext += float(e_bar @ ext[i, j] + f_now @ ins[i, j])
                if i and (i - 1, j) in mat:
                    n_open += float(e_bar[:p] @ (mat[i - 1, j] - ext[i - 1, j])) * g_a[i] * op
                if j > lo[i]:
                    n_open += float(f_now @ (mat[i, j - 1] - ins[i, j - 1])) * g_b[j] * op
                if i and j and (i - 1, j - 1) in mat:
                    v = x_bar[:p] * bm[i, j]
                    uses[i, j] = float(v @ mat[i - 1, j - 1])
                    bar[i - 1, j - 1] = bar[i - 1, j - 1] + v if (i - 1, j - 1) in bar else v
                for k in ends_at.get((i, j), ()):
                    at = (al[k] - 1, bl[k] - 1)
                    c = mat[at]
                    d_bar[k] += float(x_bar[:len(c)] @ c)
                    v = x_bar[:len(c)] * d[k]
                    bar[at] = bar[at] + v if at in bar else v
                e_here[j], f_bar = e_bar, f_now
            e_down = e_here
        return uses, d_bar, n_ext, n_open

    uses, d_bar, n_ext, n_open = back({}, True)
    prob = d * d_bar / z
    if min_am_prob > 0:
        keep = {k: d_bar[k] for k in np.nonzero(prob > math.sqrt(min_am_prob))[0].tolist()}
        bm_prob = back(keep, False)[0] / z
    else:
        bm_prob = uses / z
    out = {"log_z": np.array([math.log(z)]), "am_prob": _padded(prob, t, np.float64), "bm_prob": bm_prob}
    if grads:
        g = np.zeros(19)
        g[0], g[1] = n_ext / z / temp, n_open / z / temp
        g[2] = float(prob @ t.am_dsw) / temp
        full = uses / z
        ca, cb = np.asarray(t.code_a, int), np.asarray(t.code_b, int)
        for x in range(4):
            for y in range(4):
                g[3 + 4 * x + y] = full[np.ix_(ca == x, cb == y)].sum() / temp
        out["grads"] = g
    return out


def exact(case, seed):
    """LocARNA-P of the pairs that plain numpy does in the time there is; alignments are whole numbers."""
    if case["kind"] != "pf":
        return None
    out, spent = [], 0.0
    for t in prepare(case, seed)["tables"]:
        cost = float(t.len_a * t.len_b) ** 2  # about 4 s for one pair of 200 x 200
        if spent + cost > 5e9:
            out.append(None)
            continue
        spent += cost
        out.append(_pf_exact(t, case["min_am_prob"], case["grads"]))
    return out
