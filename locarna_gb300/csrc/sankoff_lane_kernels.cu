// The lane-per-group fill of the arc-match table D (reference:
// AlignerImpl::align_D, aligner.cc:660-732, with align_in_arcmatch :373-437 and
// align_noex :153-233 per group), for pairs without anchor constraints.
//
// A work item is up to 32 or 64 consecutive left-end groups of one pair
// (LaneItem), one or two per lane of a warp. All lanes sweep the same band cells
// (i, j), each in its own groups' matrices, so everything that depends on the
// cell alone - the base-match score, the gap costs, the list of arc matches
// ending there and their D values - is read once for all groups, the horizontal
// gap chain is a serial chain in a register instead of a warp scan, and a term
// M(a.l-1, b.l-1) + D(a, b) is one coalesced 128- or 256-byte line of the item's
// storage (line = band cell, word = group). Of the lanes' cells 40 % (60 nt) to
// 75 % (400 nt) belong to their group; the rest is outside its extent. The row sweep of run_group_c
// (sankoff_group.cuh), which gives a warp one group and its lanes the columns
// of a row, spends its instructions per group on what is shared here.
//
// Sweep order. Columns are cut into blocks of 8 and rows into quads of 4, both
// aligned to multiples; an item goes through its column blocks from left to
// right and through a block's row quads from top to bottom. In a quad (32
// cells) M of the row above and the vertical-gap state of the block's 8
// columns stay in registers; between blocks M is read back from the storage
// and the horizontal-gap state from a vector per row. An arc match spans at
// least 3 positions (a.l <= a.r - 3), so the inner corner of every term of a
// quad lies in an earlier quad of the item, and all terms of the quad are
// gathered before its cells: up to 32 entries at a time by the whole warp
// (entry, D, validity, compaction), then one line per term, 16 or 32 in
// flight, reduced into per-cell maxima of every group in shared memory. The
// entries of the quad after the next are copied to shared memory and the D
// values of the next are loaded while a quad is worked on.
//
// What bounds it, and figures (GB300, fill time): a quad is some 1,200 (32
// groups) to 1,600 (64) warp instructions behind a chain of L2 and DRAM
// latencies, 16 warps per SM; neither the issue slots (30 % used) nor DRAM (2.3 of
// 6.8 TB/s; both for 66 pairs of 180-220 nt, 64 groups) are full. 276 pairs of 60-400
// nt in two chunks: 130 ms with one warp per group, 83 ms here with 32 groups per item,
// 70 ms with 64 (fewer items to wait for, the per-quad work shared by more groups).
// Registers hold
// the rows and the loads in flight and nothing else: versions that spilled 100
// to 600 bytes took 1.3 to 2 times as long, since a spilled word comes back
// from L2 (the lines in flight leave L1 no room).
//
// States. With a gap opening go <= 0 the reference's initialisations of row al
// and column bl (init_state, aligner.cc:264-368) are what the recursion gives
// from M(al, bl) = 0 alone, so a lane only has to put a zero at its own origin
// and every cell left of or above it comes out as -inf. Cells beyond a group's
// own right ends are computed with the item's other lanes and read by nobody.
//
// Dataflow. As in sankoff_fill_kernel, items are dequeued in an order where
// producers come first and a D entry is NOT_READY until its producer's corner
// cell is final. An entry of a quad waits for a corner in the row above its
// cell at the earliest. Its producer is an earlier item, which never waits for
// a later one, or this item itself; the latter (`late` entries, by the
// producer's place in the group order) are left out of the quad's gathering,
// and such a quad goes row by row: D writes of the row above, then the row's
// late entries, then its cells.
#include <cuda_runtime.h>
#include <stdint.h>

#include "lane_sweep.cuh"
#include "sankoff_launch.hh"
#include "smem_limit.hh"

namespace lcg {

template <int GW>
__host__ __device__ inline int lane_smem_ints(int rb) {
    const int top = (smem_warp_ints(rb) + 3) & ~3;  // run_top's rows
    return top > LaneShape<GW>::SMEM ? top : LaneShape<GW>::SMEM;
}

// Terms of a quad's entries [e0, e0 + n) into the maxima, for the cells of
// `in`. The first ENTRIES entries are in shared memory at raw, their D
// values in d (all read anew with LATE). LATE: only the entries this item
// itself produces (and waits for none other), of row `row` alone; else only
// the others, of all four rows; *any_late tells whether such were left out.
// Returns the mask of cells that got a term.
template <int GW, bool LATE>
__device__ __forceinline__ unsigned lane_terms(int sb, const int *M, int raw, int cell0, int e0, int n,
                                               const int (&d)[LaneShape<GW>::STEPS], unsigned in, int row, bool *any_late) {
    const int lane = threadIdx.x & 31;
    unsigned touched = 0;
    bool late_any = false;
    for (int t0 = 0; t0 < n; t0 += LaneShape<GW>::ENTRIES) {
        const bool copied = !LATE && t0 == 0;
        const unsigned first = lc_int(sb + LaneShape<GW>::CTX, LC_FIRST), last = lc_int(sb + LaneShape<GW>::CTX, LC_LAST), shift = lc_int(sb + LaneShape<GW>::CTX, LC_SHIFT);
        const int b0 = lc_int(sb + LaneShape<GW>::CTX, LC_B0);
        int *const D = lc_ptr<int>(sb + LaneShape<GW>::CTX, LC_D);
        const int4 *const cre = lc_ptr<const int4>(sb + LaneShape<GW>::CTX, LC_CRE) + e0;
        int dv[LaneShape<GW>::STEPS];
        if (copied) {
#pragma unroll
            for (int k = 0; k < LaneShape<GW>::STEPS; ++k) dv[k] = d[k];
        } else {
            // read here: into the entries' place, D in flight together
            __syncwarp();
#pragma unroll
            for (int k = 0; k < LaneShape<GW>::STEPS; ++k) {
                const int t = t0 + 32 * k + lane;
                dv[k] = NEG;
                if (t < n) {
                    const int4 en = cre[t];
                    *(int4 *)&lcg_smem[raw + 4 * (32 * k + lane)] = en;
                    if (lane_inside(cell0, b0, en)) dv[k] = ld_volatile(D + en.x);
                }
            }
        }
        int cnt = 0;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < LaneShape<GW>::STEPS; ++k) {
            if (t0 + 32 * k >= n) break;
            const int4 en = *(const int4 *)&lcg_smem[raw + 4 * (32 * k + lane)];
            const unsigned own = __funnelshift_l(en.y, en.y, 16) + shift;
            const bool late = own <= first && own >= last;
            bool ok = t0 + 32 * k + lane < n && lane_inside(cell0, b0, en) && (in >> (en.z & 31) & 1u);
            if (LATE) ok = ok && ((en.z >> 3) & 3) == row;
            else late_any |= ok && late;
            ok = ok && late == LATE;
            int v = dv[k];
            if (ok && v == NOT_READY)
                v = wait_D(D, en.x, lc_ptr<int>(sb + LaneShape<GW>::CTX, LC_STATUS), lc_ptr<int>(sb + LaneShape<GW>::CTX, LC_ABORT));
            ok = ok && v >= MIN_FINITE;
            const unsigned mask = __ballot_sync(0xffffffffu, ok);
            touched |= __reduce_or_sync(0xffffffffu, ok ? 1u << (en.z & 31) : 0u);
            if (ok)
                *(int4 *)&lcg_smem[sb + LaneShape<GW>::STAGE + 4 * (cnt + __popc(mask & ((1u << lane) - 1)))] =
                    make_int4(((en.z >> 5) - cell0) * LaneShape<GW>::GROUPS, v, (en.z & 31) * LaneShape<GW>::GROUPS, 0);
            cnt += __popc(mask);
        }
        __syncwarp();
        // the last batch is filled up with the last term again: a maximum does not change
        const int pad = -cnt & (LaneShape<GW>::BATCH - 1);
        if (lane < pad)
            *(int4 *)&lcg_smem[sb + LaneShape<GW>::STAGE + 4 * (cnt + lane)] = *(const int4 *)&lcg_smem[sb + LaneShape<GW>::STAGE + 4 * (cnt - 1)];
        __syncwarp();
        for (int b = 0; b < cnt; b += LaneShape<GW>::BATCH) {
            typename LaneShape<GW>::Words m[LaneShape<GW>::BATCH];
            const int *const s = &lcg_smem[sb + LaneShape<GW>::STAGE + 4 * b];
#pragma unroll
            for (int u = 0; u < LaneShape<GW>::BATCH; ++u) m[u] = LaneShape<GW>::ld(M + s[4 * u]);
#pragma unroll
            for (int u = 0; u < LaneShape<GW>::BATCH; ++u) {
                const int dd = s[4 * u + 1], at = s[4 * u + 2];
#pragma unroll
                for (int v = 0; v < GW; ++v) atomicMax(&lcg_smem[sb + lane + at + 32 * v], m[u].v[v] + dd);
            }
        }
    }
    if (!LATE) *any_late = __any_sync(0xffffffffu, late_any);
    return touched;
}

// D writes of this lane's v-th group whose corner lies in quad `quad` (a
// lane_key) and, with row >= 0, in that row: fill_D_entries (aligner.cc:574-610)
// or, without lonely pairs or with stacking, the better of the corner and the
// inner arc match's own D. key: of the group's next D write, INT_MAX: none
template <int GW>
__device__ __noinline__ int lane_dwrite(int sb, const int *M, int cell0, int quad, int row, int key, int v) {
    const int lane = threadIdx.x & 31;
    const PairDev &P = *lc_ptr<const PairDev>(sb + LaneShape<GW>::CTX, LC_PAIR);
    const int4 *const rowinfo = P.rowinfo;
    int *const own = &lcg_smem[sb + LaneShape<GW>::OWN + 32 * v + lane];
    int i = own[LaneShape<GW>::GROUPS];
    while (key == quad) {
        const int4 e = P.dw[i];  // (D index, row, column, score)
        if (row >= 0 && e.y != row) break;
        const int4 ri = rowinfo[e.y];
        int x = M[(ri.w - ri.x + e.z - cell0) * LaneShape<GW>::GROUPS + v] + e.w;
        if (P.flags & (PF_NOLP | PF_STACK))
            x = max(x, inner_term<true>(P, P.dw + i, lc_ptr<int>(sb + LaneShape<GW>::CTX, LC_STATUS), lc_ptr<int>(sb + LaneShape<GW>::CTX, LC_ABORT)));
        st_volatile(P.D + e.x, norm(x));
        ++i;
        key = i < own[2 * LaneShape<GW>::GROUPS] ? lane_key(P.dw[i]) : INT_MAX;
    }
    own[LaneShape<GW>::GROUPS] = i;
    __syncwarp();
    return key;
}

template <int GW>
__device__ __forceinline__ void lane_group(const PairDev &P, const LaneItem &it, int *__restrict__ store,
                                           int *__restrict__ qrow, int sb, int *status, volatile int *abort_flag) {
    const int lane = threadIdx.x & 31;
    const int go = P.go;
    const int cell0 = P.rowinfo[it.a0].w;  // band offset of the item's first row: line 0 of the storage
    int *const M = store + lane * GW;
    const bool cls = P.flags & PF_SCLS, inner = P.flags & (PF_NOLP | PF_STACK);
    int key[GW];  // lane_key of this lane's groups' next D writes
    {
#pragma unroll
        for (int v = 0; v < GW; ++v) {
            const int k = lane * GW + v;
            int own = 0xffff, dwi = 0, dwend = 0;
            if (k < it.ng) {
                const GroupItem &g = P.groups[it.g0 + k];
                own = g.al | g.bl << 16;
                dwi = g.dw_start;
                dwend = dwi + g.dw_count;
            }
            key[v] = dwi < dwend ? lane_key(P.dw[dwi]) : INT_MAX;
            int *const o = &lcg_smem[sb + LaneShape<GW>::OWN + 32 * v + lane];
            o[0] = own;
            o[LaneShape<GW>::GROUPS] = dwi;
            o[2 * LaneShape<GW>::GROUPS] = dwend;
        }
        const GroupItem &gf = P.groups[it.g0], &gl = P.groups[it.g0 + it.ng - 1];
        if (lane == 0) {
            lc_set(sb + LaneShape<GW>::CTX, LC_CRE, P.cre);
            lc_set(sb + LaneShape<GW>::CTX, LC_D, P.D);
            lc_set(sb + LaneShape<GW>::CTX, LC_ROWINFO, P.rowinfo);
            lc_set(sb + LaneShape<GW>::CTX, LC_QSTART, P.quad_start);
            lc_set(sb + LaneShape<GW>::CTX, LC_SROW, cls ? P.rcls : P.sigma);
            lc_set(sb + LaneShape<GW>::CTX, LC_SCLS, P.scls);
            lc_set(sb + LaneShape<GW>::CTX, LC_Q, qrow);
            lc_set(sb + LaneShape<GW>::CTX, LC_STATUS, status);
            lc_set(sb + LaneShape<GW>::CTX, LC_ABORT, (const void *)abort_flag);
            lc_set(sb + LaneShape<GW>::CTX, LC_PAIR, &P);
            lc_set(sb + LaneShape<GW>::CTX, LC_BLK, P.blkrows);
            int *const c = &lcg_smem[sb + LaneShape<GW>::CTX];
            c[LC_A0] = it.a0;
            c[LC_A1] = it.a1;
            c[LC_B0] = it.b0;
            c[LC_B1] = it.b1;
            c[LC_AMAX] = it.amax;
            c[LC_FIRST] = gf.al << 16 | gf.bl;
            c[LC_LAST] = gl.al << 16 | gl.bl;
            c[LC_SHIFT] = (P.flags & PF_NOLP) ? 0x20002 : 0x10001;
            c[LC_N] = P.n;
            c[LC_M] = P.m;
            c[LC_PJ] = it.b0 >> 3;
        }
    }
#pragma unroll 8
    for (int c = 0; c < LaneShape<GW>::GROUPS; ++c) lcg_smem[sb + lane + c * 32] = NEG;
    __syncwarp();

    // two quads ahead of the sweep the entries are copied, one ahead their D
    // values and the rows' data are loaded
    lane_next_quad<GW>(sb, 0, true);
    {
        const int4 w = lane_quad<GW>(sb, 0);
        lane_prefetch<GW>(sb, sb + LaneShape<GW>::RAW, w.z, w.w);
    }
    lane_next_quad<GW>(sb, 1, false);
    {
        const int4 w = lane_quad<GW>(sb, 1);
        lane_prefetch<GW>(sb, sb + LaneShape<GW>::RAW + 4 * LaneShape<GW>::ENTRIES, w.z, w.w);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    int d[LaneShape<GW>::STEPS];
    int4 ri;     // rowinfo of row 4 q + (lane & 3)
    int sx = 0;  // row class (dense scores: row) of row 4 q + (lane >> 3)
    auto row_data = [&](int q) {
        ri = lc_ptr<const int4>(sb + LaneShape<GW>::CTX, LC_ROWINFO)[min(4 * q + (lane & 3), lc_int(sb + LaneShape<GW>::CTX, LC_N) + 1)];
        sx = min(4 * q + (lane >> 3), lc_int(sb + LaneShape<GW>::CTX, LC_N));
        if (cls) sx = lc_ptr<const int>(sb + LaneShape<GW>::CTX, LC_SROW)[sx];
    };
    {
        const int4 w = lane_quad<GW>(sb, 0);
        if (w.x < 0) return;
        lane_fetch_d<GW>(sb, store, sb + LaneShape<GW>::RAW, cell0, w.w, d);
        row_data(w.y);
    }
    int Mup[8][GW], V[8][GW];  // M and vertical-gap state max(E, M + go) of the row above
    typename LaneShape<GW>::Words Mul;             // M(i-1, j0-1)
    const typename LaneShape<GW>::Words none = [] {
        typename LaneShape<GW>::Words x;
#pragma unroll
        for (int v = 0; v < GW; ++v) x.v[v] = NEG;
        return x;
    }();
    int cs = 0, jprev = -1;
    auto dwrites = [&](int quad, int row) {
#pragma unroll
        for (int v = 0; v < GW; ++v)
            if (__any_sync(0xffffffffu, key[v] == quad)) key[v] = lane_dwrite<GW>(sb, M, cell0, quad, row, key[v], v);
    };
#pragma unroll 1
    for (int t = 0;; ++t) {
        const int4 w = lane_quad<GW>(sb, t);
        if (w.x < 0) break;
        const int J = w.x, q = w.y, i0 = q << 2, j0 = J << 3;
        if (J != jprev) {
            jprev = J;
            const int m = lc_int(sb + LaneShape<GW>::CTX, LC_M);
            if (lane < 8) lcg_smem[sb + LaneShape<GW>::GB + lane] = lc_ptr<const PairDev>(sb + LaneShape<GW>::CTX, LC_PAIR)->gapB[min(j0 + lane, m)];
            cs = min(j0 + (lane & 7), m);  // the column whose scores this lane stages
            if (cls) cs = lc_ptr<const PairDev>(sb + LaneShape<GW>::CTX, LC_PAIR)->ccls[cs];
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int v = 0; v < GW; ++v) Mup[u][v] = V[u][v] = NEG;
            Mul = none;
            if (i0 - 1 >= lc_int(sb + LaneShape<GW>::CTX, LC_A0)) {
                const int4 rp = lc_ptr<const int4>(sb + LaneShape<GW>::CTX, LC_ROWINFO)[i0 - 1];
                if (j0 - 1 >= max(lc_int(sb + LaneShape<GW>::CTX, LC_B0), rp.x) && j0 - 1 <= rp.y) Mul = LaneShape<GW>::ld(M + (rp.w - rp.x + j0 - 1 - cell0) * LaneShape<GW>::GROUPS);
            }
        }
        const int sv = cls ? lc_ptr<const int>(sb + LaneShape<GW>::CTX, LC_SCLS)[sx * 16 + cs]
                           : lc_ptr<const int>(sb + LaneShape<GW>::CTX, LC_SROW)[(size_t)sx * (lc_int(sb + LaneShape<GW>::CTX, LC_M) + 1) + cs];
        // lane r (and r + 4, ...): row i0 + r, its columns [lo, hi] in this item,
        // the line of column j0, its gap cost
        const int line = (ri.w - ri.x + j0 - cell0) * LaneShape<GW>::GROUPS, gA = ri.z;
        unsigned in, left;
        {
            int lo = INT_MAX, hi = -1;
            const int i = i0 + (lane & 3);
            if (i >= lc_int(sb + LaneShape<GW>::CTX, LC_A0) && i < lc_int(sb + LaneShape<GW>::CTX, LC_A1)) {
                lo = max(lc_int(sb + LaneShape<GW>::CTX, LC_B0), ri.x);
                hi = min(lc_int(sb + LaneShape<GW>::CTX, LC_B1) - 1, ri.y);
            }
            // the quad's cells in the item's band (bit 8 r + u), and its rows
            // whose left neighbours are (bit r)
            const unsigned in4 =
                lo <= hi && lo <= j0 + 7 && hi >= j0
                    ? (255u >> (7 - (min(hi, j0 + 7) - j0)) & 255u << (max(lo, j0) - j0)) << (8 * (lane & 3))
                    : 0u;
            in = __reduce_or_sync(0xffffffffu, in4);
            left = __ballot_sync(0xffffffffu, lo <= j0 - 1 && j0 - 1 <= hi);
        }
        // left boundary of the rows, before the terms so that its latency overlaps theirs
        int *const Q = lc_ptr<int>(sb + LaneShape<GW>::CTX, LC_Q) + i0 * LaneShape<GW>::GROUPS + lane * GW;  // horizontal-gap states of the rows before the block
        typename LaneShape<GW>::Words Ml[4], Ql[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int b = __shfl_sync(0xffffffffu, line, r);
            Ml[r] = Ql[r] = none;
            if (left >> r & 1u) {
                Ml[r] = LaneShape<GW>::ld(M + b - LaneShape<GW>::GROUPS);
                Ql[r] = LaneShape<GW>::ld(Q + r * LaneShape<GW>::GROUPS);
            }
        }
        bool any_late = false;
        unsigned touched =
            lane_terms<GW, false>(sb, M, sb + LaneShape<GW>::RAW + (t & 1) * 4 * LaneShape<GW>::ENTRIES, cell0, w.z, w.w, d, in, 0, &any_late);
        lcg_smem[sb + LaneShape<GW>::SIG + lane] = sv;
        // the next quad's D values and row data
        asm volatile("cp.async.wait_all;" ::: "memory");
        {
            const int4 x = lane_quad<GW>(sb, t + 1);
            lane_fetch_d<GW>(sb, store, sb + LaneShape<GW>::RAW + (~t & 1) * 4 * LaneShape<GW>::ENTRIES, cell0, x.w, d);
            row_data(x.x < 0 ? q : x.y);
        }
        __syncwarp();
        // D writes row by row where a row's late entries or, without lonely
        // pairs or with stacking, its own D writes read those of the row above
        const bool rowwise = any_late || inner;
        const bool starts = i0 <= lc_int(sb + LaneShape<GW>::CTX, LC_AMAX);  // groups may start in this quad
#pragma unroll 1
        for (int r = 0; r < 4; ++r) {
            const unsigned inr = in >> (8 * r);
            if (any_late) {
                const int4 x = lane_quad<GW>(sb, t);
                touched |= lane_terms<GW, true>(sb, M, sb + LaneShape<GW>::RAW + (t & 1) * 4 * LaneShape<GW>::ENTRIES, cell0, x.z, x.w, d, in,
                                            r, nullptr);
            }
            typename LaneShape<GW>::Words h = r == 0 ? Ql[0] : r == 1 ? Ql[1] : r == 2 ? Ql[2] : Ql[3], Md = Mul;
            Mul = r == 0 ? Ml[0] : r == 1 ? Ml[1] : r == 2 ? Ml[2] : Ml[3];
            int *const Mrow = M + __shfl_sync(0xffffffffu, line, r);
            const int g = __shfl_sync(0xffffffffu, gA, r);
            int start[GW];  // the origins of this lane's groups in the row
#pragma unroll
            for (int v = 0; v < GW; ++v) {
                start[v] = -1;
                if (starts) {
                    const int own = lcg_smem[sb + LaneShape<GW>::OWN + 32 * v + lane];
                    if ((own & 0xffff) == i0 + r) start[v] = (own >> 16) - j0;
                }
            }
            // Cells outside the item's band count as -inf and are not stored;
            // their gap states reach no cell inside, as the band's bounds do
            // not decrease. The maxima are >= NEG and keep M above it.
            const bool terms = touched >> (8 * r) & 255u;
#pragma unroll
            for (int c = 0; c < 8; c += 4) {
                const int4 s4 = *(const int4 *)&lcg_smem[sb + LaneShape<GW>::SIG + r * 8 + c];
                const int4 g4 = *(const int4 *)&lcg_smem[sb + LaneShape<GW>::GB + c];
                const int ss[4] = {s4.x, s4.y, s4.z, s4.w}, gb[4] = {g4.x, g4.y, g4.z, g4.w};
                int a[4][GW];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < GW; ++v) a[u][v] = NEG;
                if (terms) {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int v = 0; v < GW; ++v) {
                            int &x = lcg_smem[sb + lane + (r * 8 + c + u) * LaneShape<GW>::GROUPS + 32 * v];
                            a[u][v] = x;
                            x = NEG;
                        }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const bool ib = inr & (1u << (c + u));
                    typename LaneShape<GW>::Words X;
#pragma unroll
                    for (int v = 0; v < GW; ++v) {
                        const int E = V[c + u][v] + g;
                        const int F = h.v[v] + gb[u];
                        int x = __viaddmax_s32(Md.v[v], ss[u], __vimax3_s32(E, F, a[u][v]));
                        if (starts && c + u == start[v]) x = 0;
                        if (!ib) x = NEG;
                        V[c + u][v] = __viaddmax_s32(x, go, E);
                        h.v[v] = __viaddmax_s32(x, go, F);
                        Md.v[v] = Mup[c + u][v];
                        Mup[c + u][v] = X.v[v] = x;
                    }
                    if (ib) *(typename LaneShape<GW>::Words *)(Mrow + (c + u) * LaneShape<GW>::GROUPS) = X;
                }
            }
            if (inr & 128u) *(typename LaneShape<GW>::Words *)(Q + r * LaneShape<GW>::GROUPS) = h;
            if (rowwise) dwrites(J << 16 | q, i0 + r);
        }
        if (!rowwise) dwrites(J << 16 | q, -1);
        __syncwarp();  // the scores and entries are read before the next ones are written
        lane_next_quad<GW>(sb, (t + 2) & 3, false);
        {
            const int4 x = lane_quad<GW>(sb, t + 2);
            lane_prefetch<GW>(sb, sb + LaneShape<GW>::RAW + (t & 1) * 4 * LaneShape<GW>::ENTRIES, x.z, x.w);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// slots: per warp `slot` ints of M storage (items of pairs without kept
// rectangles) and `qslot` ints of horizontal-gap states
template <int GW, bool FAST>
__global__ void __launch_bounds__(LANE_WARPS * 32, LANE_MIN_BLOCKS)
    sankoff_lane_kernel(const PairDev *__restrict__ pairs, const int2 *__restrict__ queue, int nitems, int *scratch,
                        long long slot, long long qslot, int rb, unsigned int *qhead, int *status,
                        int *abort_flag_ptr) {
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int sbase = warp * lane_smem_ints<GW>(rb);
    int *const store = scratch + ((long long)blockIdx.x * LANE_WARPS + warp) * (slot + qslot);
    volatile int *abort_flag = abort_flag_ptr;
    while (true) {
        int idx = 0;
        if (lane == 0) idx = (int)atomicAdd(qhead, 1u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= nitems || *abort_flag) break;
        const int2 qi = queue[idx];  // (pair, item)
        const PairDev &P = pairs[qi.x];
        if (qi.y == P.nlitems) {
            run_top<false, FAST>(P, 1, sbase, rb, status, abort_flag, nullptr);
        } else {
            const LaneItem it = P.litems[qi.y];
            lane_group<GW>(P, it, P.rect ? P.rect + (long long)it.line * LaneShape<GW>::GROUPS : store, store + slot, sbase,
                       status, abort_flag);
        }
        __syncwarp();
    }
}

int lane_warps_per_block() { return LANE_WARPS; }

template <int GW>
static const void *lane_fn(bool fast) {
    return fast ? (const void *)sankoff_lane_kernel<GW, true> : (const void *)sankoff_lane_kernel<GW, false>;
}

static size_t lane_smem_bytes(int groups, int rb) {
    return (size_t)LANE_WARPS * sizeof(int) * (groups == 64 ? lane_smem_ints<2>(rb) : lane_smem_ints<1>(rb));
}

cudaError_t lane_occupancy(int groups, int rb, bool fast, int *blocks_per_sm) {
    const size_t smem = lane_smem_bytes(groups, rb);
    const void *fn = groups == 64 ? lane_fn<2>(fast) : lane_fn<1>(fast);
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    *blocks_per_sm = 0;
    if (smem > (size_t)optin) return cudaSuccess;
    e = allow_smem(fn, smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, LANE_WARPS * 32, smem);
}

cudaError_t launch_lane_fill(int groups, const PairDev *pairs, const int2 *queue, int nitems, int *scratch,
                             long long slot, long long qslot, int rb, bool fast, unsigned int *qhead, int *status,
                             int *abort_flag, int blocks, cudaStream_t st) {
    const size_t smem = lane_smem_bytes(groups, rb);
    auto *const fn = groups == 64 ? (fast ? sankoff_lane_kernel<2, true> : sankoff_lane_kernel<2, false>)
                                  : (fast ? sankoff_lane_kernel<1, true> : sankoff_lane_kernel<1, false>);
    fn<<<blocks, LANE_WARPS * 32, smem, st>>>(pairs, queue, nitems, scratch, slot, qslot, rb, qhead, status,
                                              abort_flag);
    return cudaGetLastError();
}

}  // namespace lcg
