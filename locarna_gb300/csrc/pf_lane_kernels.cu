// LocARNA-P in FP32 with 32 left-end groups per warp, one per lane: the inside
// pass and its adjoint (the recursions are in pf_kernels.cu, which gives a warp
// one group; the sweep by column blocks and row quads, its storage of one line
// per band cell and the dataflow are those of sankoff_lane_kernels.cu).
//
// All lanes sweep the same cells, so the gap chains are serial chains in
// registers instead of warp scans, a cell's weights and a quad's entries are
// read once for 32 groups, and an arc match's uses are counted per item instead
// of per group. Cells above or left of a group's origin have M = 0 and carry
// nothing; cells beyond its right ends get values nobody reads and have the
// adjoint 0, as no seed lies behind them.
//
// The adjoint goes through the quads in reverse. In a quad, in this order:
// - the seeds: D_bar w of the D entries whose corner is in the quad into M_bar,
//   once every use of the entry has been back-propagated (the counters);
// - the cells, rows from the bottom, columns from the right; X_bar of each cell
//   and its base-match sum's term X_bar bm M(i-1,j-1) go to shared memory;
// - the entries: X_bar s D into M_bar of the corner's line (a reduction in L2,
//   32 words wide), X_bar s M(corner) summed over the lanes into D_bar, then the
//   counters drop, after one fence per quad.
// A use lies at (a.r, b.r), the seed at (a.r-1, b.r-1): earlier in this order,
// or, if both are in one quad and of one item, a row below; such quads go row by
// row. An item waits only for items that come before it.
//
// Sums over lanes are taken by one lane per cell or entry over its 32 words in
// shared memory, with next to no rounding (pfl_row_sum), so that they are as good
// as the FP64 atomics over single groups they replace; they end in FP64 atomics, 32
// times fewer.
//
// What bounds it, and figures (GB300): a warp's serial chain of quads, each some
// 10,000 cycles backward, half of them latency of L2 and DRAM, and the waits for
// the uses behind it; issue slots are a quarter used, DRAM at 1.5 of 6.8 TB/s.
// Backward over 28 pairs of 160-200 nt: 23 ms with one warp per group, 9.7 here (M kept
// by the forward pass); 21 pairs of 80-500 nt: 123 and 48.5; forward 5.1 and 4.9, 32 and
// 26. M swept again: 66 pairs of 280-320 nt 333 and 271. What mattered on the way: an entry's
// lines copied to shared memory in one go (21 pairs: 104 -> 50 ms; loads behind a
// branch came one by one), no register spilled (64 loads in flight with 460 bytes
// spilled: 57 instead of 50), and one copy of the entries' code (57 -> 46: a second
// one for row by row did not fit the instruction cache). In the forward pass
// joining the two copies cost more than it saved (25.5 -> 26.3).
#include <cuda_runtime.h>

#include <algorithm>

#include "lane_sweep.cuh"
#include "pf_sweep.cuh"
#include "smem_limit.hh"

namespace lcg {

using PL = LaneShape<1>;
constexpr int PFL_SUMS = PL::SMEM;  // backward: what is summed over lanes, [cell or entry][group]
constexpr int PFL_FWD_INTS = PL::SMEM, PFL_BACK_INTS = PL::SMEM + 1024;
static_assert(LANE_WARPS == PF_WARPS, "one block shape");

__device__ __forceinline__ float &pfl_f(int i) { return ((float *)lcg_smem)[i]; }

// What the lanes share (LaneWord) and the lane's group: its left ends and its D
// writes [first, past the last one) in PL::OWN
__device__ __forceinline__ void pfl_context(const PFPair<float> &P, const LaneItem &it, float *qrow, int sb, int *status,
                                            volatile int *abort_flag) {
    const int lane = threadIdx.x & 31;
    int own = 0xffff, first = 0, end = 0;
    if (lane < it.ng) {
        const GroupItem &g = P.groups[it.g0 + lane];
        own = g.al | g.bl << 16;
        first = g.dw_start;
        end = first + g.dw_count;
    }
    int *const o = &lcg_smem[sb + PL::OWN + lane];
    o[0] = own;
    o[PL::GROUPS] = first;
    o[2 * PL::GROUPS] = end;
    const GroupItem &gf = P.groups[it.g0], &gl = P.groups[it.g0 + it.ng - 1];
    const int cx = sb + PL::CTX;
    if (lane == 0) {
        lc_set(cx, LC_CRE, P.cre);
        lc_set(cx, LC_D, P.D);
        lc_set(cx, LC_ROWINFO, P.rowinfo);
        lc_set(cx, LC_QSTART, P.quad_start);
        lc_set(cx, LC_SROW, P.bm);
        lc_set(cx, LC_SCLS, P.gA);
        lc_set(cx, LC_Q, qrow);
        lc_set(cx, LC_STATUS, status);
        lc_set(cx, LC_ABORT, (const void *)abort_flag);
        lc_set(cx, LC_PAIR, &P);
        lc_set(cx, LC_BLK, P.blkrows);
        int *const c = &lcg_smem[cx];
        c[LC_A0] = it.a0;
        c[LC_A1] = it.a1;
        c[LC_B0] = it.b0;
        c[LC_B1] = it.b1;
        c[LC_AMAX] = it.amax;
        c[LC_FIRST] = gf.al << 16 | gf.bl;
        c[LC_LAST] = gl.al << 16 | gl.bl;
        c[LC_SHIFT] = 0x10001;
        c[LC_N] = P.n;
        c[LC_M] = P.m;
        c[LC_PJ] = it.b0 >> 3;
    }
#pragma unroll 8
    for (int c = 0; c < 32; ++c) lcg_smem[sb + lane + c * 32] = 0;
    __syncwarp();
}

// whether an entry's producer is a group of the item
__device__ __forceinline__ bool pfl_own(int cx, int4 en) {
    const unsigned own = __funnelshift_l(en.y, en.y, 16) + (unsigned)lc_int(cx, LC_SHIFT);
    return own <= (unsigned)lc_int(cx, LC_FIRST) && own >= (unsigned)lc_int(cx, LC_LAST);
}

// 8 floats from shared memory (16-byte aligned)
__device__ __forceinline__ void pfl_load8(int at, float (&v)[8]) {
#pragma unroll
    for (int c = 0; c < 8; c += 4) {
        const float4 x = *(const float4 *)&lcg_smem[at + c];
        v[c] = x.x;
        v[c + 1] = x.y;
        v[c + 2] = x.z;
        v[c + 3] = x.w;
    }
}

// The sum of the words [first, last) (multiples of PFL_PART) of row `row` of PFL_SUMS
// in one thread, PFL_PART at a time. Every word is split without error into multiples
// of a unit that the largest one sets, of a unit 2^18 times smaller, and a remainder
// (vector extraction; Rump, Ogita, Oishi 2008): with top < 2^(e + 1) the units are
// 2^(e - 17) and 2^(e - 35), so that up to 32 of the parts add up exactly in FP32, and
// only the remainders, below 2^(e - 35), are rounded. That is better than a sum in
// FP64, of which an SM adds two a clock. Backward of 21 pairs of 80-500 nt: 48.5 ms; a
// two-sum per word (2^-43 off) 46.1; of 66 pairs of 280-320 nt, whose M is swept again,
// 271 and 273. All 32 words in straight-line code cost the latter 292 (instruction
// cache), parts of 8 cost the former 51.
constexpr int PFL_PART = 16;
__device__ __noinline__ double pfl_row_sum(int sb, int row, int first, int last) {
    const int at = sb + PFL_SUMS + 32 * row;
    double sum = 0.0;
#pragma unroll 1
    for (int k = first; k < last; k += PFL_PART) {
        float x[PFL_PART], top = 0.f;
#pragma unroll
        for (int t = 0; t < PFL_PART; ++t) {
            x[t] = pfl_f(at + ((row + k + t) & 31));  // (lanes on different banks)
            top = fmaxf(top, fabsf(x[t]));
        }
        const int ex = __float_as_int(top) >> 23;
        if (top != 0.f && (ex < 27 || ex > 227)) {
            // the units would leave FP32's range (or an infinity)
#pragma unroll 1
            for (int t = 0; t < PFL_PART; ++t) sum += (double)pfl_f(at + ((row + k + t) & 31));
            continue;
        }
        const float c0 = __int_as_float((ex + 6) << 23) * 1.5f, c1 = c0 * 0x1p-18f;
        float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int t = 0; t < PFL_PART; ++t) {
            const float a = (x[t] + c0) - c0, y = x[t] - a, b = (y + c1) - c1;
            s0 += a;
            s1 += b;
            s2 += y - b;
        }
        sum += (double)s0 + ((double)s1 + (double)s2);
    }
    return sum;
}

// the sums of rows [0, n), lane k that of row k: two lanes a row where that is enough
__device__ __forceinline__ double pfl_row_sums(int sb, int n) {
    const int lane = threadIdx.x & 31;
    const bool two = n <= 16;
    const int row = two ? lane & 15 : lane, first = two ? lane & 16 : 0;
    double v = row < n ? pfl_row_sum(sb, row, first, two ? first + 16 : 32) : 0.0;
    if (two) v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
}

// ---------------------------------------------------------------- forward

// Terms M(corner) D of a quad's entries [e0, e0 + n) into the sums at RAW of
// PL, as lane_terms takes their maxima. PRODUCE: the forward pass - waits for D,
// counts the uses and leaves the item's own entries to LATE; else D is final.
template <bool LATE, bool PRODUCE>
__device__ __forceinline__ unsigned pfl_terms(int sb, const float *M, int raw, int cell0, int e0, int n,
                                              const int (&d)[PL::STEPS], unsigned in, int row, bool *any_late) {
    const int lane = threadIdx.x & 31, cx = sb + PL::CTX;
    unsigned touched = 0;
    bool late_any = false;
    for (int t0 = 0; t0 < n; t0 += PL::ENTRIES) {
        const int b0 = lc_int(cx, LC_B0);
        const int *const D = lc_ptr<const int>(cx, LC_D);
        int dv[PL::STEPS];
        if (!LATE && t0 == 0) {
#pragma unroll
            for (int k = 0; k < PL::STEPS; ++k) dv[k] = d[k];
        } else {
            const int4 *const cre = lc_ptr<const int4>(cx, LC_CRE) + e0;
            __syncwarp();
#pragma unroll
            for (int k = 0; k < PL::STEPS; ++k) {
                const int t = t0 + 32 * k + lane;
                dv[k] = 0;
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
        for (int k = 0; k < PL::STEPS; ++k) {
            if (t0 + 32 * k >= n) break;
            const int4 en = *(const int4 *)&lcg_smem[raw + 4 * (32 * k + lane)];
            bool ok = t0 + 32 * k + lane < n && lane_inside(cell0, b0, en) && (in >> (en.z & 31) & 1u);
            if (PRODUCE) {
                const bool late = pfl_own(cx, en);
                if (LATE) ok = ok && ((en.z >> 3) & 3) == row;
                else late_any |= ok && late;
                ok = ok && late == LATE;
            }
            int v = dv[k];
            if (PRODUCE && ok && v == PF_NOT_READY_F32)
                v = __float_as_int(pf_wait((const float *)D + en.x, lc_ptr<int>(cx, LC_STATUS), lc_ptr<int>(cx, LC_ABORT)));
            ok = ok && v != 0;
            if (PRODUCE && ok) atomicAdd(lc_ptr<const PFPair<float>>(cx, LC_PAIR)->cnt + en.x, 1);
            const unsigned mask = __ballot_sync(0xffffffffu, ok);
            touched |= __reduce_or_sync(0xffffffffu, ok ? 1u << (en.z & 31) : 0u);
            if (ok)
                *(int4 *)&lcg_smem[sb + PL::STAGE + 4 * (cnt + __popc(mask & ((1u << lane) - 1)))] =
                    make_int4(((en.z >> 5) - cell0) * 32, v, (en.z & 31) * 32, 0);
            cnt += __popc(mask);
        }
        __syncwarp();
        // the last batch is filled up with the last term again, of weight 0
        const int pad = -cnt & (PL::BATCH - 1);
        if (lane < pad) {
            int4 s = *(const int4 *)&lcg_smem[sb + PL::STAGE + 4 * (cnt - 1)];
            s.y = 0;
            *(int4 *)&lcg_smem[sb + PL::STAGE + 4 * (cnt + lane)] = s;
        }
        __syncwarp();
        // entries come by cells: a cell's sum is kept in a register
        float acc = 0.f;
        int cur = -1;
        for (int b = 0; b < cnt; b += PL::BATCH) {
            float m[PL::BATCH];
            const int *const s = &lcg_smem[sb + PL::STAGE + 4 * b];
#pragma unroll
            for (int u = 0; u < PL::BATCH; ++u) m[u] = M[s[4 * u]];
#pragma unroll
            for (int u = 0; u < PL::BATCH; ++u) {
                const int at = s[4 * u + 2];
                if (at != cur) {
                    if (cur >= 0) pfl_f(sb + lane + cur) += acc;
                    acc = 0.f;
                    cur = at;
                }
                acc = fmaf(m[u], __int_as_float(s[4 * u + 1]), acc);
            }
        }
        if (cur >= 0) pfl_f(sb + lane + cur) += acc;
    }
    if (!LATE) *any_late = __any_sync(0xffffffffu, late_any);
    return touched;
}

// D writes of the lane's group whose corner lies in quad `quad` (a lane_key)
// and, with row >= 0, in that row. key: of its next D write, INT_MAX: none
__device__ __noinline__ int pfl_dwrite(int sb, const float *M, int cell0, int quad, int row, int key) {
    const PFPair<float> &P = *lc_ptr<const PFPair<float>>(sb + PL::CTX, LC_PAIR);
    int *const own = &lcg_smem[sb + PL::OWN + (threadIdx.x & 31)];
    int i = own[PL::GROUPS];
    while (key == quad) {
        const int4 e = P.dw[i];  // (D index, row, column, -)
        if (row >= 0 && e.y != row) break;
        const int4 ri = P.rowinfo[e.y];
        *(volatile float *)(P.D + e.x) = M[(ri.w - ri.x + e.z - cell0) * 32] * P.w[e.x];
        ++i;
        key = i < own[2 * PL::GROUPS] ? lane_key(P.dw[i]) : INT_MAX;
    }
    own[PL::GROUPS] = i;
    __syncwarp();
    return key;
}

// The inside sweep of an item (lane_group): M to `store`, one line per band
// cell. PRODUCE: the forward pass; else only M is wanted and D is final.
template <bool PRODUCE>
__device__ __forceinline__ void pfl_sweep(const PFPair<float> &P, const LaneItem &it, float *__restrict__ store,
                                          float *__restrict__ qrow, int sb, int *status, volatile int *abort_flag) {
    const int lane = threadIdx.x & 31, cx = sb + PL::CTX;
    const float o = P.o, inv_s = P.inv_s, arcf = P.arcf;
    const int cell0 = P.rowinfo[it.a0].w;
    float *const M = store + lane;
    pfl_context(P, it, qrow, sb, status, abort_flag);
    int key = INT_MAX;
    if (PRODUCE) {
        const int *const own = &lcg_smem[sb + PL::OWN + lane];
        if (own[PL::GROUPS] < own[2 * PL::GROUPS]) key = lane_key(P.dw[own[PL::GROUPS]]);
    }
    lane_next_quad<1>(sb, 0, true);
    {
        const int4 w = lane_quad<1>(sb, 0);
        lane_prefetch<1>(sb, sb + PL::RAW, w.z, w.w);
    }
    lane_next_quad<1>(sb, 1, false);
    {
        const int4 w = lane_quad<1>(sb, 1);
        lane_prefetch<1>(sb, sb + PL::RAW + 4 * PL::ENTRIES, w.z, w.w);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    int d[PL::STEPS];
    int4 ri;      // rowinfo of row 4 q + (lane & 3)
    float gA;     // its gap weight
    int sx = 0;   // the row whose base-match weights the lane stages: 4 q + (lane >> 3)
    auto row_data = [&](int q) {
        const int n = lc_int(cx, LC_N), i = 4 * q + (lane & 3);
        ri = lc_ptr<const int4>(cx, LC_ROWINFO)[min(i, n + 1)];
        gA = lc_ptr<const float>(cx, LC_SCLS)[min(i, n)];
        sx = min(4 * q + (lane >> 3), n);
    };
    {
        const int4 w = lane_quad<1>(sb, 0);
        if (w.x < 0) return;
        lane_fetch_d<1>(sb, (const int *)store, sb + PL::RAW, cell0, w.w, d);
        row_data(w.y);
    }
    float Mup[8], V[8];  // M of the row above, and E + o N there (its vertical-gap state)
    float Mul = 0.f;     // M(i-1, j0-1)
    int cs = 0, jprev = -1;
    auto dwrites = [&](int quad, int row) {
        if (PRODUCE && __any_sync(0xffffffffu, key == quad)) key = pfl_dwrite(sb, M, cell0, quad, row, key);
    };
#pragma unroll 1
    for (int t = 0;; ++t) {
        const int4 w = lane_quad<1>(sb, t);
        if (w.x < 0) break;
        const int J = w.x, q = w.y, i0 = q << 2, j0 = J << 3;
        if (J != jprev) {
            jprev = J;
            const int m = lc_int(cx, LC_M);
            if (lane < 8)
                pfl_f(sb + PL::GB + lane) = lc_ptr<const PFPair<float>>(cx, LC_PAIR)->gB[min(j0 + lane, m)];
            cs = min(j0 + (lane & 7), m);
#pragma unroll
            for (int u = 0; u < 8; ++u) Mup[u] = V[u] = 0.f;
            Mul = 0.f;
            if (i0 - 1 >= lc_int(cx, LC_A0)) {
                const int4 rp = lc_ptr<const int4>(cx, LC_ROWINFO)[i0 - 1];
                if (j0 - 1 >= max(lc_int(cx, LC_B0), rp.x) && j0 - 1 <= rp.y) Mul = M[(rp.w - rp.x + j0 - 1 - cell0) * 32];
            }
        }
        const float sv = lc_ptr<const float>(cx, LC_SROW)[(size_t)sx * (lc_int(cx, LC_M) + 1) + cs];
        const int line = (ri.w - ri.x + j0 - cell0) * 32;
        unsigned in, left;
        {
            int lo = INT_MAX, hi = -1;
            const int i = i0 + (lane & 3);
            if (i >= lc_int(cx, LC_A0) && i < lc_int(cx, LC_A1)) {
                lo = max(lc_int(cx, LC_B0), ri.x);
                hi = min(lc_int(cx, LC_B1) - 1, ri.y);
            }
            const unsigned in4 =
                lo <= hi && lo <= j0 + 7 && hi >= j0
                    ? (255u >> (7 - (min(hi, j0 + 7) - j0)) & 255u << (max(lo, j0) - j0)) << (8 * (lane & 3))
                    : 0u;
            in = __reduce_or_sync(0xffffffffu, in4);
            left = __ballot_sync(0xffffffffu, lo <= j0 - 1 && j0 - 1 <= hi);
        }
        const float gAv = gA;
        float *const Q = lc_ptr<float>(cx, LC_Q) + i0 * 32 + lane;  // F + o Q of the rows' cells before the block
        float Ml[4], Ql[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int b = __shfl_sync(0xffffffffu, line, r);
            Ml[r] = Ql[r] = 0.f;
            if (left >> r & 1u) {
                Ml[r] = M[b - 32];
                Ql[r] = Q[r * 32];
            }
        }
        bool any_late = false;
        unsigned touched = pfl_terms<false, PRODUCE>(sb, M, sb + PL::RAW + (t & 1) * 4 * PL::ENTRIES, cell0, w.z, w.w, d,
                                                     in, 0, &any_late);
        pfl_f(sb + PL::SIG + lane) = sv;
        asm volatile("cp.async.wait_all;" ::: "memory");
        {
            const int4 x = lane_quad<1>(sb, t + 1);
            lane_fetch_d<1>(sb, (const int *)store, sb + PL::RAW + (~t & 1) * 4 * PL::ENTRIES, cell0, x.w, d);
            row_data(x.x < 0 ? q : x.y);
        }
        __syncwarp();
        const bool starts = i0 <= lc_int(cx, LC_AMAX);  // groups may start in this quad
#pragma unroll 1
        for (int r = 0; r < 4; ++r) {
            const unsigned inr = in >> (8 * r);
            if (any_late) {
                const int4 x = lane_quad<1>(sb, t);
                touched |= pfl_terms<true, PRODUCE>(sb, M, sb + PL::RAW + (t & 1) * 4 * PL::ENTRIES, cell0, x.z, x.w, d,
                                                    in, r, nullptr);
            }
            float h = r == 0 ? Ql[0] : r == 1 ? Ql[1] : r == 2 ? Ql[2] : Ql[3], Md = Mul;
            Mul = r == 0 ? Ml[0] : r == 1 ? Ml[1] : r == 2 ? Ml[2] : Ml[3];
            float *const Mrow = M + __shfl_sync(0xffffffffu, line, r);
            const float g = __shfl_sync(0xffffffffu, gAv, r);
            int start = -1;  // the origin of the lane's group in the row
            if (starts) {
                const int own = lcg_smem[sb + PL::OWN + lane];
                if ((own & 0xffff) == i0 + r) start = (own >> 16) - j0;
            }
            // Cells outside the item's band count as 0; their gap states reach
            // no cell inside, as the band's bounds do not decrease.
            float ss[8], gb[8], a[8];  // (read before anything is written: a store would hold up the loads)
            pfl_load8(sb + PL::SIG + r * 8, ss);
            pfl_load8(sb + PL::GB, gb);
            const bool terms = touched >> (8 * r) & 255u;
#pragma unroll
            for (int u = 0; u < 8; ++u) a[u] = terms ? pfl_f(sb + lane + (r * 8 + u) * 32) : 0.f;
            if (terms)
#pragma unroll
                for (int u = 0; u < 8; ++u) pfl_f(sb + lane + (r * 8 + u) * 32) = 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const bool ib = inr & (1u << u);
                float X = fmaf(a[u], arcf, Md * ss[u]);
                float E = V[u] * g, F = h * gb[u];
                if (starts && u == start) X = inv_s;
                if (!ib) X = E = F = 0.f;
                const float N = X + F, Mx = N + E;
                V[u] = fmaf(o, N, E);
                h = fmaf(o, X + E, F);
                Md = Mup[u];
                Mup[u] = Mx;
                if (ib) Mrow[u * 32] = Mx;
            }
            if (inr & 128u) Q[r * 32] = h;
            if (any_late) dwrites(J << 16 | q, i0 + r);
        }
        if (!any_late) dwrites(J << 16 | q, -1);
        __syncwarp();  // the weights and entries are read before the next ones are written
        lane_next_quad<1>(sb, (t + 2) & 3, false);
        {
            const int4 x = lane_quad<1>(sb, t + 2);
            lane_prefetch<1>(sb, sb + PL::RAW + (t & 1) * 4 * PL::ENTRIES, x.z, x.w);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// ---------------------------------------------------------------- backward

// 16 bytes to shared memory, zeros without `from` (src is then not read)
__device__ __forceinline__ void pfl_copy16(int dst, const float *src, bool from) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(&lcg_smem[dst]);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(from ? 16 : 0) : "memory");
}

// lane_next_quad in the reverse order: blocks from the right, quads from the bottom
__device__ __forceinline__ void pfl_prev_quad(int sb, int slot, bool first) {
    const int cx = sb + PL::CTX;
    int J = lc_int(cx, LC_PJ), q = lc_int(cx, LC_PQ), qa = lc_int(cx, LC_PQB), k = lc_int(cx, LC_PK);
    __syncwarp();
    if (J >= 0 && !first && q > qa) {
        --q;
        --k;
    } else if (J >= 0) {
        const int last = lc_int(cx, LC_B0) >> 3;
        J = first ? (lc_int(cx, LC_B1) - 1) >> 3 : J - 1;
        for (;; --J) {
            if (J < last) {
                J = -1;
                break;
            }
            const int4 b = lc_ptr<const int4>(cx, LC_BLK)[J];
            qa = max(b.x, lc_int(cx, LC_A0) >> 2);
            q = min(b.y, (lc_int(cx, LC_A1) - 1) >> 2);
            k = b.z + q - b.x;
            if (q >= qa) break;  // (blocks the band reaches below the item's rows only are left out)
        }
    }
    int e = 0, n = 0;
    if (J >= 0) {
        const int *const qs = lc_ptr<const int>(cx, LC_QSTART);
        e = qs[k];
        n = qs[k + 1] - e;
    }
    if ((threadIdx.x & 31) == 0) {
        *(int4 *)&lcg_smem[sb + PL::QUAD + 4 * slot] = make_int4(J, q, e, n);
        int *const c = &lcg_smem[cx];
        c[LC_PJ] = J;
        c[LC_PQ] = q;
        c[LC_PQB] = qa;
        c[LC_PK] = k;
    }
    __syncwarp();
}

// The lane's seeds in quad `quad` and, with row >= 0, in that row: D_bar w into
// M_bar of the corner, which is in shared memory by then. key: of the group's last D write not seeded yet, -1: none
template <bool TRUNC>
__device__ __noinline__ int pfl_seed(int sb, int quad, int row, int key, double theta_z) {
    const int cx = sb + PL::CTX;
    const PFPair<float> &P = *lc_ptr<const PFPair<float>>(cx, LC_PAIR);
    int *const own = &lcg_smem[sb + PL::OWN + (threadIdx.x & 31)];
    int i = own[2 * PL::GROUPS] - 1;
    while (key == quad) {
        const int4 e = P.dw[i];
        if (row >= 0 && e.y != row) break;
        bool seed = true;
        if (TRUNC) {
            seed = (double)P.D[e.x] * P.Dbar[e.x] > theta_z;
        } else {
            volatile int *const abort_flag = lc_ptr<int>(cx, LC_ABORT);
            long long spins = 0;
            while (*(const volatile int *)(P.cnt + e.x) > 0) {
                __nanosleep(64);
                if (++spins > PF_SPIN_LIMIT || *abort_flag) {
                    atomicOr(lc_ptr<int>(cx, LC_STATUS), ST_TIMEOUT);
                    *abort_flag = 1;
                    break;
                }
            }
            __threadfence();
        }
        if (seed)
            pfl_f(sb + (threadIdx.x & 31) + 32 * ((e.y & 3) * 8 + (e.z & 7))) += (float)ld_cg(P.Dbar + e.x) * P.w[e.x];
        --i;
        key = i >= own[PL::GROUPS] ? lane_key(P.dw[i]) : -1;
    }
    own[2 * PL::GROUPS] = i + 1;
    __syncwarp();
    return key;
}

// whether a quad has entries that the item itself produces (not if all its
// groups have one left end of A: a use lies inside)
__device__ __forceinline__ bool pfl_any_late(int sb, int raw, int cell0, int e0, int n, unsigned in) {
    const int lane = threadIdx.x & 31, cx = sb + PL::CTX;
    const int b0 = lc_int(cx, LC_B0);
    bool late = false;
    for (int t = lane; t < n; t += 32) {
        const int4 en = t < PL::ENTRIES ? *(const int4 *)&lcg_smem[raw + 4 * t] : lc_ptr<const int4>(cx, LC_CRE)[e0 + t];
        late |= lane_inside(cell0, b0, en) && (in >> (en.z & 31) & 1u) && pfl_own(cx, en);
    }
    return __any_sync(0xffffffffu, late);
}

// The entries of a quad (row >= 0: of that row alone) on the way back. nz: the
// cells where some lane's X_bar is not 0
template <bool TRUNC>
__device__ __forceinline__ void pfl_back_terms(int sb, const float *store, float *Mb, int raw, int cell0, int e0, int n,
                                               const int (&d)[PL::STEPS], unsigned in, unsigned nz, int row) {
    const int lane = threadIdx.x & 31, cx = sb + PL::CTX;
    for (int t0 = 0; t0 < n; t0 += PL::ENTRIES) {
        const int b0 = lc_int(cx, LC_B0);
        int dv[PL::STEPS];
        if (row < 0 && t0 == 0) {
#pragma unroll
            for (int k = 0; k < PL::STEPS; ++k) dv[k] = d[k];
        } else {
            const int4 *const cre = lc_ptr<const int4>(cx, LC_CRE) + e0;
            const int *const D = lc_ptr<const int>(cx, LC_D);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < PL::STEPS; ++k) {
                const int t = t0 + 32 * k + lane;
                dv[k] = 0;
                if (t < n) {
                    const int4 en = cre[t];
                    *(int4 *)&lcg_smem[raw + 4 * (32 * k + lane)] = en;
                    if (lane_inside(cell0, b0, en)) dv[k] = ld_volatile(D + en.x);
                }
            }
        }
        __syncwarp();
        const PFPair<float> &P = *lc_ptr<const PFPair<float>>(cx, LC_PAIR);
        int cnt = 0;
        unsigned uses = 0;  // bit k: the lane's entry of step k is used by the item
#pragma unroll
        for (int k = 0; k < PL::STEPS; ++k) {
            if (t0 + 32 * k >= n) break;
            const int4 en = *(const int4 *)&lcg_smem[raw + 4 * (32 * k + lane)];
            bool ok = t0 + 32 * k + lane < n && lane_inside(cell0, b0, en) && (in >> (en.z & 31) & 1u) && dv[k] != 0;
            if (row >= 0) ok = ok && ((en.z >> 3) & 3) == row;
            if (ok) uses |= 1u << k;
            ok = ok && (nz >> (en.z & 31) & 1u);
            const unsigned mask = __ballot_sync(0xffffffffu, ok);
            if (ok)
                *(int4 *)&lcg_smem[sb + PL::STAGE + 4 * (cnt + __popc(mask & ((1u << lane) - 1)))] =
                    make_int4(((en.z >> 5) - cell0) * 32, dv[k], (en.z & 31) * 32, en.x);
            cnt += __popc(mask);
        }
        __syncwarp();
        // filled up to a multiple of 16 with the last entry again, of weight 0
        const int pad = -cnt & 15;
        if (lane < pad) {
            int4 x = *(const int4 *)&lcg_smem[sb + PL::STAGE + 4 * (cnt - 1)];
            x.y = 0;
            *(int4 *)&lcg_smem[sb + PL::STAGE + 4 * (cnt + lane)] = x;
        }
        __syncwarp();
        const float arcf = P.arcf;
        for (int b = 0; b < cnt; b += 32) {
            const int nb = min(32, cnt - b), np = nb > 16 ? 32 : 16;
            const int *const s = &lcg_smem[sb + PL::STAGE + 4 * b];
            if (!TRUNC) {
                // M of the corners to where the terms will be
                for (int k = lane >> 3; k < np; k += 4)
                    pfl_copy16(sb + PFL_SUMS + 32 * k + 4 * (lane & 7), store + s[4 * k] + 4 * (lane & 7), true);
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
            }
#pragma unroll 1
            for (int h = 0; h < np; h += 8) {
                int4 e[8];
                float x[8], p[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) e[u] = *(const int4 *)&s[4 * (h + u)];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    x[u] = pfl_f(sb + lane + e[u].z) * arcf;
                    if (!TRUNC) p[u] = pfl_f(sb + PFL_SUMS + 32 * (h + u) + lane);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float y = x[u] * __int_as_float(e[u].y);
                    if (y != 0.f) atomicAdd(Mb + e[u].x, y);
                    if (!TRUNC) pfl_f(sb + PFL_SUMS + 32 * (h + u) + lane) = x[u] != 0.f ? x[u] * p[u] : 0.f;
                }
            }
            if (!TRUNC) {
                __syncwarp();
                const double sum = pfl_row_sums(sb, nb);
                if (lane < nb) atomicAdd(P.Dbar + s[4 * lane + 3], sum);
                __syncwarp();
            }
        }
        // the D_bar updates are visible before the counters drop, those of M_bar
        // before other lanes copy its lines
        if (TRUNC && cnt > 0) __threadfence();
        if (!TRUNC && __any_sync(0xffffffffu, uses != 0)) {
            __threadfence();
            __syncwarp();
#pragma unroll
            for (int k = 0; k < PL::STEPS; ++k)
                if (uses >> k & 1u) atomicSub(P.cnt + lcg_smem[raw + 4 * (32 * k + lane)], 1);
        }
        __syncwarp();
    }
}

// The adjoint of pfl_sweep on its M in `store`: M_bar in `bstore`, a line per
// band cell; qrow: per row two lines, gB F_bar and X_bar bm of the first cell of
// the block to the right.
template <bool TRUNC>
__device__ __forceinline__ void pfl_back(const PFPair<float> &P, const LaneItem &it, const float *__restrict__ store,
                                         float *bstore, float *qrow, int sb, int *status, volatile int *abort_flag,
                                         double theta_z) {
    const int lane = threadIdx.x & 31, cx = sb + PL::CTX;
    const float o = P.o;
    const int cell0 = P.rowinfo[it.a0].w;
    {
        float4 *const z = (float4 *)bstore;
        const int nz4 = (P.rowinfo[it.a1].w - cell0) * 8;
        for (int k = lane; k < nz4; k += 32) z[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __threadfence();  // (and M where this warp has just written it: lanes copy each other's words)
    const float *const M = store + lane;
    float *const Mb = bstore + lane;
    pfl_context(P, it, qrow, sb, status, abort_flag);
    int key = -1;
    {
        const int *const own = &lcg_smem[sb + PL::OWN + lane];
        if (own[PL::GROUPS] < own[2 * PL::GROUPS]) key = lane_key(P.dw[own[2 * PL::GROUPS] - 1]);
    }
    pfl_prev_quad(sb, 0, true);
    {
        const int4 w = lane_quad<1>(sb, 0);
        lane_prefetch<1>(sb, sb + PL::RAW, w.z, w.w);
    }
    pfl_prev_quad(sb, 1, false);
    {
        const int4 w = lane_quad<1>(sb, 1);
        lane_prefetch<1>(sb, sb + PL::RAW + 4 * PL::ENTRIES, w.z, w.w);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    int d[PL::STEPS];
    int4 ri;     // rowinfo of row 4 q - 1 + (lane & 7)
    float gA;    // its gap weight
    int sx = 0;  // the row whose base-match weights the lane stages
    auto row_data = [&](int q) {
        const int n = lc_int(cx, LC_N), i = max(4 * q - 1 + (lane & 7), 0);
        ri = lc_ptr<const int4>(cx, LC_ROWINFO)[min(i, n + 1)];
        gA = lc_ptr<const float>(cx, LC_SCLS)[min(i, n)];
        sx = min(4 * q + (lane >> 3), n);
    };
    {
        const int4 w = lane_quad<1>(sb, 0);
        if (w.x < 0) return;
        lane_fetch_d<1>(sb, (const int *)store, sb + PL::RAW, cell0, w.w, d);
        row_data(w.y);
    }
    float U[8], Dd[8];  // of the row below: gA E_bar, and X_bar bm of the cell to the right
    float below = 0.f;  // the latter of the block's last column
    int cs = 0, jprev = -1;
    unsigned cm = 0;  // columns of the block right of the lane's origin
    auto seeds = [&](int quad, int row) {
        if (__any_sync(0xffffffffu, key == quad)) key = pfl_seed<TRUNC>(sb, quad, row, key, theta_z);
    };
#pragma unroll 1
    for (int t = 0;; ++t) {
        const int4 w = lane_quad<1>(sb, t);
        if (w.x < 0) break;
        const int J = w.x, q = w.y, i0 = q << 2, j0 = J << 3;
        const int raw = sb + PL::RAW + (t & 1) * 4 * PL::ENTRIES;
        const bool entered = J != jprev;
        if (entered) {
            jprev = J;
            const int m = lc_int(cx, LC_M);
            if (lane < 8)
                pfl_f(sb + PL::GB + lane) = lc_ptr<const PFPair<float>>(cx, LC_PAIR)->gB[min(j0 + lane, m)];
            cs = min(j0 + (lane & 7), m);
#pragma unroll
            for (int u = 0; u < 8; ++u) U[u] = Dd[u] = 0.f;
            const int b = (lcg_smem[sb + PL::OWN + lane] >> 16) - j0;  // columns up to b are not right of it
            cm = b < 0 ? 255u : b >= 7 ? 0u : 255u << (b + 1) & 255u;
        }
        pfl_f(sb + PL::SIG + lane) = lc_ptr<const float>(cx, LC_SROW)[(size_t)sx * (lc_int(cx, LC_M) + 1) + cs];
        // lane l < 6: row i0 - 1 + l, the line of column j0, and which of the
        // columns j0 - 1 .. j0 + 8 the item's band has there
        const int line = (ri.w - ri.x + j0 - cell0) * 32;
        const float gAv = gA;
        unsigned m10 = 0;
        {
            const int i = i0 - 1 + lane;
            if (lane < 6 && i >= lc_int(cx, LC_A0) && i < lc_int(cx, LC_A1)) {
                const int lo = max(max(lc_int(cx, LC_B0), ri.x) - (j0 - 1), 0);
                const int hi = min(min(lc_int(cx, LC_B1) - 1, ri.y) - (j0 - 1), 9);
                if (lo <= hi) m10 = ((2u << (hi - lo)) - 1) << lo;
            }
        }
        const unsigned in =
            __reduce_or_sync(0xffffffffu, lane >= 1 && lane <= 4 ? (m10 >> 1 & 255u) << (8 * (lane - 1)) : 0u);
        if (entered)
            below = __shfl_sync(0xffffffffu, m10, 5) >> 9 & 1u ? lc_ptr<float>(cx, LC_Q)[(i0 + 4) * 64 + 32 + lane] : 0.f;
        // M_bar of the quad's cells and M of their upper left neighbours to where
        // X_bar and the base-match terms will be (row by row the latter are read
        // again with the rows, as the entries' sums take their place)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int r = k >> 1, u = (k & 1) * 4 + (lane >> 3), at = (4 * k + (lane >> 3)) * 32 + 4 * (lane & 7);
            const unsigned mC = __shfl_sync(0xffffffffu, m10, r + 1), mU = __shfl_sync(0xffffffffu, m10, r);
            const int lC = __shfl_sync(0xffffffffu, line, r + 1), lU = __shfl_sync(0xffffffffu, line, r);
            pfl_copy16(sb + at, bstore + lC + u * 32 + 4 * (lane & 7), mC >> (u + 1) & 1u);
            pfl_copy16(sb + PFL_SUMS + at, store + lU + (u - 1) * 32 + 4 * (lane & 7), mU >> u & 1u);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        const bool rowwise = !TRUNC && it.amax > it.a0 && pfl_any_late(sb, raw, cell0, w.z, w.w, in);
        unsigned nzl = 0;  // the lane's cells with X_bar not 0
        const int al = lcg_smem[sb + PL::OWN + lane] & 0xffff;
#pragma unroll 1
        for (int r = 3; r >= 0; --r) {
            const int i = i0 + r;
            if (rowwise || r == 3) seeds(J << 16 | q, rowwise ? i : -1);
            const unsigned mC = __shfl_sync(0xffffffffu, m10, r + 1);
            const float g = __shfl_sync(0xffffffffu, gAv, r + 1);
            float *const Q = lc_ptr<float>(cx, LC_Q) + i * 64 + lane;
            if (rowwise) {
                const unsigned mU = __shfl_sync(0xffffffffu, m10, r);
                const float *const Mu = M + __shfl_sync(0xffffffffu, line, r) - 32;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    pfl_f(sb + PFL_SUMS + lane + (r * 8 + u) * 32) = mU >> u & 1u ? Mu[u * 32] : 0.f;
            }
            float hb = 0.f;  // gB F_bar of the cell to the right
            Dd[7] = below;
            below = 0.f;
            if (mC >> 9 & 1u) {
                hb = Q[0];
                below = Q[32];
            }
            const unsigned act = i > al ? mC >> 1 & cm : 0u;
            float right = 0.f;  // X_bar bm of the cell to the right
            float ss[8], gb[8], mb[8], md[8];  // (read before anything is written)
            pfl_load8(sb + PL::SIG + r * 8, ss);
            pfl_load8(sb + PL::GB, gb);
            const int at = sb + lane + r * 256;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                mb[u] = pfl_f(at + u * 32);
                md[u] = pfl_f(at + PFL_SUMS + u * 32);
            }
#pragma unroll
            for (int u = 7; u >= 0; --u) {
                const float mbar = mb[u] + Dd[u];
                const float MN = fmaf(U[u], o, mbar), Qb = hb * o;
                float F = hb + MN, E = mbar + (Qb + U[u]), X = MN + Qb;
                if (!(act >> u & 1u)) F = E = X = 0.f;
                if (u < 7) Dd[u] = right;
                hb = F * gb[u];
                U[u] = E * g;
                right = X * ss[u];
                mb[u] = X;
                md[u] = right != 0.f ? right * md[u] : 0.f;
                if (X != 0.f) nzl |= 1u << (r * 8 + u);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                pfl_f(at + u * 32) = mb[u];
                pfl_f(at + PFL_SUMS + u * 32) = md[u];
            }
            if (mC >> 1 & 1u) {
                Q[0] = hb;
                Q[32] = right;
            }
            // (one place each for the seeds, the sums and the entries, row by
            // row or not: a second copy of that code is felt in the instruction cache)
            if (rowwise || r == 0) {
                const unsigned nz = __reduce_or_sync(0xffffffffu, nzl), cells = rowwise ? nz & 255u << (8 * r) : nz;
                // the base-match sums
                const int at = (__shfl_sync(0xffffffffu, line, (lane >> 3) + 1) >> 5) + cell0 + (lane & 7);
                __syncwarp();
                if (cells >> lane & 1u)
                    atomicAdd(lc_ptr<const PFPair<float>>(cx, LC_PAIR)->bmacc + at, pfl_row_sum(sb, lane, 0, 32));
                __syncwarp();
                pfl_back_terms<TRUNC>(sb, store, Mb, raw, cell0, w.z, w.w, d, in, nz, rowwise ? r : -1);
            }
        }
        // the next quad's D values and rows, the one's after it entries
        {
            const int4 x = lane_quad<1>(sb, t + 1);
            lane_fetch_d<1>(sb, (const int *)store, sb + PL::RAW + (~t & 1) * 4 * PL::ENTRIES, cell0, x.w, d);
            row_data(x.x < 0 ? q : x.y);
        }
        __syncwarp();
        pfl_prev_quad(sb, (t + 2) & 3, false);
        {
            const int4 x = lane_quad<1>(sb, t + 2);
            lane_prefetch<1>(sb, raw, x.z, x.w);
        }
        {
            // the next quad's lines on the way to L2
            const int4 x = lane_quad<1>(sb, t + 1);
            const int l = (lane >> 3) + 1, i = 4 * x.y + (lane >> 3), j = 8 * x.x + (lane & 7);
            const int rx = __shfl_sync(0xffffffffu, ri.x, l), ry = __shfl_sync(0xffffffffu, ri.y, l);
            const int rw = __shfl_sync(0xffffffffu, ri.w, l);
            if (x.x >= 0 && i >= lc_int(cx, LC_A0) && i < lc_int(cx, LC_A1) && j >= rx && j <= ry) {
                const int at = (rw - rx + j - cell0) * 32;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(bstore + at));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(store + at));
            }
        }
        if (*abort_flag) break;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// ---------------------------------------------------------------- kernels

// slots: `block` floats of scratch per block; per warp `slot` of them for M
// where the pairs have no kept storage, then the vectors per row (backward:
// `slot` for M_bar first)
__global__ void __launch_bounds__(LANE_WARPS * 32, LANE_MIN_BLOCKS)
    pf_lane_fwd_kernel(const PFPair<float> *__restrict__ pairs, int npairs, const int2 *__restrict__ queue, int nitems,
                       float *scratch, long long block, long long slot, long long warp_floats, int rb,
                       unsigned int *qhead, unsigned int *topq, int *status, int *abort_ptr) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sb = warp * PFL_FWD_INTS;
    float *const mine = scratch + blockIdx.x * block + warp * warp_floats;
    volatile int *abort_flag = abort_ptr;
    while (true) {
        int idx = 0;
        if (lane == 0) idx = (int)atomicAdd(qhead, 1u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= nitems || *abort_flag) break;
        const int2 qi = queue[idx];  // (pair, item)
        const PFPair<float> &P = pairs[qi.x];
        const LaneItem it = P.litems[qi.y];
        pfl_sweep<true>(P, it, P.rect ? P.rect + (long long)it.line * 32 : mine, mine + slot, sb, status, abort_flag);
        __syncwarp();
    }
    __shared__ float sm[2][2 * PF_WARPS];
    for (int q; (q = pf_next_top(topq, npairs, abort_flag)) < npairs;) {
        const PFPair<float> &P = pairs[q];
        pf_top_sweep<float, true, true, false>(P, nullptr, nullptr, pf_rows<float>(0, rb), sm, status, abort_flag);
        if (threadIdx.x == 0) P.res[0] = log((double)P.topM[(size_t)P.n * (P.m + 1) + P.m]);
    }
}

template <bool TRUNC>
__global__ void __launch_bounds__(LANE_WARPS * 32, LANE_MIN_BLOCKS)
    pf_lane_back_kernel(const PFPair<float> *__restrict__ pairs, int npairs, const int2 *__restrict__ queue, int nitems,
                        float *scratch, long long block, long long slot, long long back_slot, long long warp_floats,
                        int rb, unsigned int *qhead, unsigned int *topq, int *status, int *abort_ptr, double theta) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *abort_flag = abort_ptr;
    {
        __shared__ float sm[2][2 * PF_WARPS];
        for (int q; (q = pf_next_top(topq, npairs, abort_flag)) < npairs;)
            pf_top_back<float, TRUNC, false>(pairs[q], pairs[q].topM, nullptr, nullptr, scratch + blockIdx.x * block,
                                             pf_rows<float>(0, rb), sm, nullptr, nullptr);
    }
    const int sb = warp * PFL_BACK_INTS;
    float *const mine = scratch + blockIdx.x * block + warp * warp_floats;
    while (true) {
        int idx = 0;
        if (lane == 0) idx = (int)atomicAdd(qhead, 1u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= nitems || *abort_flag) break;
        const int2 qi = queue[nitems - 1 - idx];  // the consumers of an item's D entries come first
        const PFPair<float> &P = pairs[qi.x];
        const LaneItem it = P.litems[qi.y];
        const double theta_z = TRUNC ? theta * exp(P.res[0]) : 0.0;
        if (TRUNC) {
            // an item none of whose arc matches passes the threshold contributes nothing
            bool any = false;
            if (lane < it.ng) {
                const GroupItem &g = P.groups[it.g0 + lane];
                for (int k = 0; k < g.dw_count && !any; ++k) {
                    const int pos = P.dw[g.dw_start + k].x;
                    any = (double)P.D[pos] * P.Dbar[pos] > theta_z;
                }
            }
            if (!__any_sync(0xffffffffu, any)) continue;
        }
        float *const qrow = mine + slot + back_slot;
        const float *store = mine;
        if (P.rect) store = P.rect + (long long)it.line * 32;
        else pfl_sweep<false>(P, it, mine, qrow, sb, status, abort_flag);
        pfl_back<TRUNC>(P, it, store, mine + slot, qrow, sb, status, abort_flag, theta_z);
        __syncwarp();
    }
}

// ---------------------------------------------------------------- launchers

static size_t pfl_smem(bool back, int rb) {
    const size_t rows = sizeof(float) * PF_RING_ROWS * (size_t)rb;  // the top level's
    return std::max(rows, sizeof(int) * LANE_WARPS * (size_t)(back ? PFL_BACK_INTS : PFL_FWD_INTS));
}

static cudaError_t pfl_occupancy(const void *fn, size_t smem, int *blocks_per_sm) {
    cudaError_t e = allow_smem(fn, smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, LANE_WARPS * 32, smem);
}

cudaError_t pf_lane_occupancy(int rb, int *blocks_per_sm) {
    int f = 0, b = 0, c = 0;
    cudaError_t e = pfl_occupancy((const void *)pf_lane_fwd_kernel, pfl_smem(false, rb), &f);
    if (e == cudaSuccess) e = pfl_occupancy((const void *)pf_lane_back_kernel<false>, pfl_smem(true, rb), &b);
    if (e == cudaSuccess) e = pfl_occupancy((const void *)pf_lane_back_kernel<true>, pfl_smem(true, rb), &c);
    *blocks_per_sm = std::min(f, std::min(b, c));
    return e;
}

cudaError_t pf_launch_lane_fwd(const void *pairs, int npairs, const int2 *queue, int nitems, const PFLaneScratch &s, int rb,
                               unsigned int *qhead, unsigned int *topq, int *status, int *abort_flag, cudaStream_t st) {
    pf_lane_fwd_kernel<<<s.blocks, LANE_WARPS * 32, pfl_smem(false, rb), st>>>(
        (const PFPair<float> *)pairs, npairs, queue, nitems, (float *)s.base, s.block, s.slot, s.warp, rb, qhead, topq,
        status, abort_flag);
    return cudaGetLastError();
}

cudaError_t pf_launch_lane_back(const void *pairs, int npairs, const int2 *queue, int nitems, const PFLaneScratch &s,
                                int rb, unsigned int *qhead, unsigned int *topq, int *status, int *abort_flag,
                                cudaStream_t st, double theta) {
    auto k = theta > 0.0 ? pf_lane_back_kernel<true> : pf_lane_back_kernel<false>;
    k<<<s.blocks, LANE_WARPS * 32, pfl_smem(true, rb), st>>>((const PFPair<float> *)pairs, npairs, queue, nitems,
                                                             (float *)s.base, s.block, s.slot, s.back_slot, s.warp, rb,
                                                             qhead, topq, status, abort_flag, theta);
    return cudaGetLastError();
}

}  // namespace lcg
