// What the lane-per-group sweeps share (sankoff_lane_kernels.cu, where the
// sweep is described, and pf_lane_kernels.cu): the layout of a warp's shared
// memory, the walk over an item's quads and the copies ahead of it.
#pragma once
#include <cuda_runtime.h>

#include "sankoff_group.cuh"

namespace lcg {

constexpr int LANE_WARPS = 4;        // warps per block
constexpr int LANE_MIN_BLOCKS = 4;   // 128 registers a thread: more would spill

// GW groups per lane
template <int GW>
struct LaneShape {
    static constexpr int GROUPS = 32 * GW;
    static constexpr int BATCH = GW == 1 ? 32 : 16;  // term lines in flight per warp
    static constexpr int STEPS = GW == 1 ? 3 : 2;    // batches of 32 entries staged together
    static constexpr int ENTRIES = 32 * STEPS;
    // Shared ints per warp (offsets from its base): the maxima of a quad's cells
    // [cell][group], the first ENTRIES entries of two quads (copied ahead), the
    // staged terms (int4, padded to a full batch), the quad's base-match scores,
    // the block's gap costs, the descriptors of four quads (J, q, first entry,
    // entries), what the lanes share (LC_*), and per group its left ends and D
    // writes (al | bl << 16, the next one, past the last one). A group's place:
    // word v of lane l's GW in the storage (l GW + v), v * 32 + l in shared memory.
    static constexpr int RAW = 32 * GROUPS;
    static constexpr int STAGE = RAW + 2 * 4 * ENTRIES;
    static constexpr int SIG = STAGE + 4 * ENTRIES;
    static constexpr int GB = SIG + 32;
    static constexpr int QUAD = GB + 8;
    static constexpr int CTX = QUAD + 16;
    static constexpr int OWN = CTX + 40;
    static constexpr int SMEM = OWN + 3 * GROUPS;
    static_assert(SMEM % 4 == 0, "16-byte rows");
    static_assert(ENTRIES % BATCH == 0, "padding stays inside the stage");
    struct alignas(4 * GW) Words {  // one lane's groups
        int v[GW];
    };
    __device__ static __forceinline__ Words ld(const int *p) { return *(const Words *)p; }
};
// the sweep's registers are for its matrix rows and loads in flight: everything
// read once a quad is kept in shared memory (a register spill comes back from
// L2, the lines in flight having emptied L1)
enum LaneWord {
    LC_CRE = 0, LC_D = 2, LC_ROWINFO = 4, LC_QSTART = 6, LC_SROW = 8, LC_SCLS = 10, LC_Q = 12, LC_STATUS = 14,
    LC_ABORT = 16, LC_PAIR = 18, LC_BLK = 20,  // pointers
    LC_A0 = 22, LC_A1, LC_B0, LC_B1, LC_AMAX, LC_FIRST, LC_LAST, LC_SHIFT, LC_N, LC_M,
    LC_PJ, LC_PQ, LC_PQB, LC_PK                // the quad whose entries are copied next
};

// cx: lcg_smem offset of the shared words
__device__ __forceinline__ int lc_int(int cx, int k) { return *(volatile int *)&lcg_smem[cx + k]; }
template <typename T>
__device__ __forceinline__ T *lc_ptr(int cx, int k) {
    return (T *)*(volatile unsigned long long *)&lcg_smem[cx + k];
}
__device__ __forceinline__ void lc_set(int cx, int k, const void *p) {
    *(unsigned long long *)&lcg_smem[cx + k] = (unsigned long long)p;
}

__device__ __forceinline__ void lane_copy16(int dst, const void *src) {  // dst: lcg_smem offset
    const unsigned d = (unsigned)__cvta_generic_to_shared(&lcg_smem[dst]);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// Copy the first ENTRIES entries [e, e + n) of a quad to shared memory; each lane reads its own copies
template <int GW>
__device__ __forceinline__ void lane_prefetch(int sb, int raw, int e, int n) {
    const int lane = threadIdx.x & 31;
    const int4 *const src = lc_ptr<const int4>(sb + LaneShape<GW>::CTX, LC_CRE) + e;
#pragma unroll
    for (int k = 0; k < LaneShape<GW>::STEPS; ++k)
        if (32 * k + lane < n) lane_copy16(raw + 4 * (32 * k + lane), src + 32 * k + lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// whether an entry's corner lies in the item's storage, by rows and by columns
__device__ __forceinline__ bool lane_inside(int cell0, int b0, int4 en) {
    return en.z >> 5 >= cell0 && en.y >> 16 >= b0;  // (a corner outside the band has cell 0)
}

// D of the copied entries (NOT_READY where still to be written), loads in
// flight on return. At 32 groups an item the lines of their terms (store: line
// 0) are sent for as well: 24 pairs of 80-130 nt 3.59 -> 3.43 ms, 12 of
// 180-220 nt 6.53 -> 6.18; at 64 groups 9 pairs of 300-400 nt took 23.2 -> 23.3.
template <int GW>
__device__ __forceinline__ void lane_fetch_d(int sb, const int *store, int raw, int cell0, int n,
                                             int (&d)[LaneShape<GW>::STEPS]) {
    const int lane = threadIdx.x & 31;
    const int *const D = lc_ptr<const int>(sb + LaneShape<GW>::CTX, LC_D);
    const int b0 = lc_int(sb + LaneShape<GW>::CTX, LC_B0);
#pragma unroll
    for (int k = 0; k < LaneShape<GW>::STEPS; ++k) {
        d[k] = NEG;
        if (32 * k + lane < n) {
            const int4 en = *(const int4 *)&lcg_smem[raw + 4 * (32 * k + lane)];
            if (lane_inside(cell0, b0, en)) {
                d[k] = ld_volatile(D + en.x);
                if (GW == 1)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(store + ((en.z >> 5) - cell0) * 32));
            }
        }
    }
}

// where a D write's corner comes in the sweep: its column block and row quad
__device__ __forceinline__ int lane_key(int4 e) { return (e.z >> 3) << 16 | e.y >> 2; }

// Move the prefetch position to the item's next quad in sweep order (first:
// to its first quad) and write that quad's descriptor; past the last one, a
// descriptor with block -1.
template <int GW>
__device__ __forceinline__ void lane_next_quad(int sb, int slot, bool first) {
    int J = lc_int(sb + LaneShape<GW>::CTX, LC_PJ), q = lc_int(sb + LaneShape<GW>::CTX, LC_PQ), qb = lc_int(sb + LaneShape<GW>::CTX, LC_PQB), k = lc_int(sb + LaneShape<GW>::CTX, LC_PK);
    __syncwarp();
    if (J >= 0 && !first && q < qb) {
        ++q;
        ++k;
    } else if (J >= 0) {
        if (!first) ++J;
        if (J > (lc_int(sb + LaneShape<GW>::CTX, LC_B1) - 1) >> 3) {
            J = -1;
        } else {
            // the quads whose rows' bands meet the block, the index of the first
            const int4 b = lc_ptr<const int4>(sb + LaneShape<GW>::CTX, LC_BLK)[J];
            q = max(b.x, lc_int(sb + LaneShape<GW>::CTX, LC_A0) >> 2);
            qb = min(b.y, (lc_int(sb + LaneShape<GW>::CTX, LC_A1) - 1) >> 2);
            k = b.z + q - b.x;
            if (q > qb) J = -1;  // the band has left the item's rows
        }
    }
    int e = 0, n = 0;
    if (J >= 0) {
        const int *const qs = lc_ptr<const int>(sb + LaneShape<GW>::CTX, LC_QSTART);
        e = qs[k];
        n = qs[k + 1] - e;
    }
    if ((threadIdx.x & 31) == 0) {
        *(int4 *)&lcg_smem[sb + LaneShape<GW>::QUAD + 4 * slot] = make_int4(J, q, e, n);
        int *const c = &lcg_smem[sb + LaneShape<GW>::CTX];
        c[LC_PJ] = J;
        c[LC_PQ] = q;
        c[LC_PQB] = qb;
        c[LC_PK] = k;
    }
    __syncwarp();
}

template <int GW>
__device__ __forceinline__ int4 lane_quad(int sb, int slot) {
    return *(const int4 *)&lcg_smem[sb + LaneShape<GW>::QUAD + 4 * (slot & 3)];
}

}  // namespace lcg
