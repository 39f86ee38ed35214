// The index structures of a pair that hold something per arc match, made on the
// device from the arc matches in ArcMatches order (what engine.cu's prep_pair
// makes on the host for other orders): the candidate lists by row (crow) and by
// cell of the right ends (cre), the D entries, the D writes of every left-end
// group and, with stacking, the inner arc matches. Reference: ArcMatches,
// arc_matches.cc:19-188; lex_greater_left_ends, arc_matches.hh:188-220.
//
// The order of the input makes every list an ordered scatter: arcs of A come by
// left end descending, arc matches of one arc by left end of B descending, so
// the arc matches of the arcs that end in a row, taken in index order, are the
// row's list, and those of a cell among them the cell's list in the order that
// the traceback wants. One warp per row (and per left end of A) goes through
// them 32 at a time; within 32, arc matches of the same cell (group) are ranked
// with a match of the warp's lanes, and a cursor per cell (group) carries on.
//
// Bound by the latency of a row's few hundred entries, not by its bytes (8 read
// and 60 written per arc match): both kernels take 0.1 ms for the 120,000 arc
// matches of a 400 x 400 pair, whose host preparation fell from 5.3 to 1.8 ms;
// 276 pairs of 60-400 nt (4 M arc matches per chunk): host preparation 46 to 15
// ms, packing 7.6 to 4.9 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include "index_device.cuh"

namespace lcg {

constexpr int INDEX_WARPS = 8;

__device__ __forceinline__ bool ix_in_band(const PairDev &P, int i, int j) {
    return P.min_col[i] <= j && j <= P.max_col[i];
}

// rank of this lane among the lanes of `all` with the same value, and whether it is the last of them
__device__ __forceinline__ int ix_rank(unsigned all, int value, bool *last) {
    const unsigned same = __match_any_sync(all, value);
    const int lane = threadIdx.x & 31;
    *last = (same >> lane) == 1u;
    return __popc(same & ((1u << lane) - 1));
}

// crow, cre, am_pos and D of row i
__global__ void __launch_bounds__(INDEX_WARPS * 32)
    index_rows_kernel(const PairDev *__restrict__ pairs, const IndexPair *__restrict__ ix) {
    const PairDev &P = pairs[blockIdx.x];
    const IndexPair &X = ix[blockIdx.x];
    const int i = blockIdx.y * INDEX_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (!X.arcs || i > P.n) return;
    const int lo = P.min_col[i], hi = P.max_col[i];
    const int4 ri = P.rowinfo[i];
    const int cell0 = ri.w - lo;
    int2 *const crow = (int2 *)P.crow;
    int4 *const cre = (int4 *)P.cre;
    for (int j = lo + lane; j <= hi; j += 32) X.cursor[cell0 + j] = P.cre_start[cell0 + j];
    __syncwarp();
    int pos0 = P.rowarc[i].x;
    for (int s = X.row_start[i]; s < X.row_start[i + 1]; ++s) {
        const int4 a = X.arcs[X.row_arcs[s]];  // (l, r, first and past its last arc match)
        const int al1 = a.x - 1;
        const int4 rc = P.rowinfo[al1];  // the row of the inner corners
        for (int k0 = a.z; k0 < a.w; k0 += 32) {
            const int k = k0 + lane;
            const int lr = k < a.w ? X.am_lr[k] : 0;
            const int bl = lr & 0xffff, br = lr >> 16;
            const bool ok = k < a.w && br >= lo && br <= hi;
            const unsigned mask = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const int pos = pos0 + __popc(mask & ((1u << lane) - 1));
                bool last;
                const int at = X.cursor[cell0 + br] + ix_rank(mask, br, &last);
                __syncwarp(mask);
                if (last) X.cursor[cell0 + br] = at + 1;
                const bool corner = rc.x <= bl - 1 && bl - 1 <= rc.y;
                const unsigned cc = corner ? rc.w + bl - 1 - rc.x : 0;
                crow[pos] = make_int2(al1 | ((bl - 1) << 16), br);
                cre[at] = make_int4(pos, al1 | ((bl - 1) << 16), (int)(cc << 5 | (i & 3) << 3 | (br & 7)), k);
                // written by the group of its left ends, if there is one and its corner is in the band
                const bool group = ix_in_band(P, a.x, bl) && corner && a_match(P, a.x, bl) && ix_in_band(P, i - 1, br - 1);
                P.D[pos] = group ? NOT_READY : NEG;
                X.am_pos[k] = pos;
            } else if (k < a.w) {
                X.am_pos[k] = -1;
            }
            pos0 += __popc(mask);
            __syncwarp();
        }
    }
}

// The D writes of the groups of one left end of A, their arc matches' kept
// rectangles and, with stacking, inner arc matches
__global__ void __launch_bounds__(INDEX_WARPS * 32)
    index_groups_kernel(const PairDev *__restrict__ pairs, const IndexPair *__restrict__ ix) {
    const PairDev &P = pairs[blockIdx.x];
    const IndexPair &X = ix[blockIdx.x];
    const int w = blockIdx.y * INDEX_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (!X.arcs || w >= X.nlefts) return;
    const int4 left = X.lefts[w];  // (first and past its last arc, first and past its last group)
    int4 *const dw = (int4 *)P.dw;
    int2 *const dwn = (int2 *)P.dwn;
    const bool lanes = P.flags & PF_LANES, stack = (P.flags & PF_STACK) && X.inner_a;
    for (int g = left.z + lane; g < left.w; g += 32) X.gcursor[g] = P.groups[g].dw_start;
    __syncwarp();
    for (int s = left.x; s < left.y; ++s) {
        const int4 a = X.arcs[s];
        for (int k0 = a.z; k0 < a.w; k0 += 32) {
            const int k = k0 + lane;
            const bool on = k < a.w;
            const int lr = on ? X.am_lr[k] : 0;
            const int bl = lr & 0xffff, br = lr >> 16;
            // its group: bl descends over the left end's groups
            int x = left.z, y = left.w;
            while (x < y) {
                const int c = (x + y) / 2;
                if (P.groups[c].bl > bl) x = c + 1;
                else y = c;
            }
            const bool group = on && x < left.w && P.groups[x].bl == bl;
            const int pos = on ? X.am_pos[k] : -1;
            if (on && P.am_rect) {
                int2 rect = lanes ? make_int2(0, -1) : make_int2(-1, 0);
                if (group && lanes) {
                    const LaneItem it = P.litems[x / P.lane_groups];
                    rect = make_int2(it.line - P.rowinfo[it.a0].w, x % P.lane_groups);
                } else if (group && P.groups[x].rect_off >= 0) {
                    rect = make_int2(P.groups[x].rect_off, P.groups[x].br - bl);
                }
                ((int2 *)P.am_rect)[k] = rect;
            }
            int2 inner = make_int2(-1, -1);
            if (on && stack) {
                // (l + 1, r - 1) of both arcs: the first arc match of that pair of arcs
                const int ia = X.inner_a[s], ib = X.inner_b[X.am_b[k]];
                if (ia >= 0 && ib >= 0) {
                    int u = X.arcs[ia].z, v = X.arcs[ia].w;
                    while (u < v) {
                        const int c = (u + v) / 2;
                        if (X.am_b[c] < ib) u = c + 1;
                        else v = c;
                    }
                    if (u < X.arcs[ia].w && X.am_b[u] == ib) inner = make_int2(u, X.am_pos[u]);
                }
                ((int2 *)P.inner)[k] = inner;
            }
            const bool ok = group && pos >= 0 && ix_in_band(P, a.y - 1, br - 1);
            const unsigned mask = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                bool last;
                const int at = X.gcursor[x] + ix_rank(mask, x, &last);
                __syncwarp(mask);
                if (last) X.gcursor[x] = at + 1;
                dw[at] = make_int4(pos, a.y - 1, br - 1, P.am_score[k]);
                if (stack) {
                    const bool st = inner.x >= 0 && X.am_stackable[k];
                    dwn[at] = st ? make_int2(inner.y, P.am_sscore[k]) : make_int2(-1, 0);
                }
            }
            __syncwarp();
        }
    }
    if (!lanes) return;  // index order is by right end of A: the row order
    // lane per group: by column block, then row, the order of that sweep
    for (int g = left.z + lane; g < left.w; g += 32) {
        const int d0 = P.groups[g].dw_start, d1 = d0 + P.groups[g].dw_count;
        for (int u = d0 + 1; u < d1; ++u) {
            const int4 e = dw[u];
            const int2 f = stack ? dwn[u] : make_int2(0, 0);
            const int key = (e.z >> 3) << 16 | e.y;
            int v = u;
            for (; v > d0 && ((dw[v - 1].z >> 3) << 16 | dw[v - 1].y) > key; --v) {
                dw[v] = dw[v - 1];
                if (stack) dwn[v] = dwn[v - 1];
            }
            dw[v] = e;
            if (stack) dwn[v] = f;
        }
    }
}

cudaError_t launch_index(const PairDev *pairs, const IndexPair *ix, int npairs, int max_n, int max_lefts,
                         cudaStream_t st) {
    const int rows = (max_n + INDEX_WARPS) / INDEX_WARPS;
    index_rows_kernel<<<dim3(npairs, rows), INDEX_WARPS * 32, 0, st>>>(pairs, ix);
    const int lefts = (max_lefts + INDEX_WARPS - 1) / INDEX_WARPS;
    if (lefts > 0) index_groups_kernel<<<dim3(npairs, lefts), INDEX_WARPS * 32, 0, st>>>(pairs, ix);
    return cudaGetLastError();
}

}  // namespace lcg
