// Device-side records of the LocARNA-P engine shared by the kernels
// (pf_kernels.cu) and the host side (engine_pf.cu).
#pragma once
#include <cuda_runtime.h>

#include "lcg_device.cuh"

namespace lcg {

// NOT_READY pattern of a D entry that a group has yet to write (a NaN that no
// arithmetic produces).
constexpr long long PF_NOT_READY_F64 = 0x7ff4c0de00000000ll;
constexpr int PF_NOT_READY_F32 = 0x7fa0c0de;

template <typename T>
struct PFPair {
    int n, m;
    int num_am;
    const int4 *rowinfo;   // n+2: (min_col, max_col, -, band offset)
    const int2 *crow;      // ((a.l-1) | (b.l-1) << 16, b.r) by row a.r, a.l descending
    const int2 *rowarc;    // n+2: [start, end) of row i's entries in crow
    const T *bm;           // (n+1)(m+1) scaled base-match weights
    const T *gA, *gB;      // scaled gap weights
    T o;                   // gap-opening weight
    T gu;                  // the value of every gB[j], j >= 1, if they are all the same, else 0; 0 in FP32 with gap gradients
    const T *gpow;         // 33: its powers 0 to 32, each rounded once
    T inv_s;               // 1 / pf_scale
    T arcf;                // pf_scale / c^4
    // per D position (the arc match's position in crow):
    const T *w;            // arc-match weight
    T *D;                  // NOT_READY pattern until written
    double *Dbar;          // dZ'/dD (backward), accumulated in FP64
    int *cnt;              // number of uses still to be back-propagated
    // the top level, (n+1)(m+1) each, with zeros around the band: M, and E and F
    // (nullptr: not kept; only the gap gradients read them)
    T *topM, *topE, *topF;
    double *bmacc;         // per band cell (row offset rowinfo.w): sum of X_bar M(i-1,j-1) bm, FP64
    double *res;           // [0] log Z', [1] gap-extension uses, [2] gap-opening uses
    const GroupItem *groups;  // left-end groups (work items) in dependency order (then the top level)
    const int4 *dw;           // D writes: (D index, ar-1, br-1, -), by group, ar ascending
    // Kept group rectangles (nullptr: the backward recomputes them): the
    // forward writes group g's M (rect_states 1) or M, E, F (3; the gap
    // gradients read E and F) to rect + rect_states g.rect_off, state k at
    // k (ar-al)(br-bl), row i-al, column j-bl, pitch br-bl; the backward
    // reads them instead of recomputing the group.
    T *rect;
    int rect_states;
    // Pairs swept lane per group (FP32, pf_lane_kernels.cu): the work items and
    // the entries by quad as in PairDev; dw is then ordered by column block and
    // row, rect holds the items' kept storage (a line of 32 per band cell)
    const LaneItem *litems;
    const int4 *cre;
    const int4 *blkrows;
    const int *quad_start;
};

// A pair's arc matches, in the caller's order, and its results
struct PFArcMatches {
    int na, bandcells;
    const int *score;   // per arc match
    const double *dsw;  // its derivative by the structure weight (nullptr: no offset of that)
    const int *pos;     // its D index, -1: never a term
    const int *D0;      // per D index: NOT_READY if a group writes it
    double *prob;
    double zs;          // Z in the scaled frame
};

// Scratch of the lane-per-group launches, in floats: per block, in it per warp,
// in that for M (0: kept) and, backward, for M_bar; then the vectors per row
struct PFLaneScratch {
    void *base = nullptr;
    long long block = 0, warp = 0, slot = 0, back_slot = 0;
    int blocks = 0;
};

// queue: (pair, group) work items in dependency-respecting order, the top
// levels apart (topq counts those taken); keep_states: 0, or the pairs'
// PFPair::rect_states (rectangles kept); top_ef: PFPair::topE and topF are set
template <typename T>
cudaError_t pf_launch_fwd(const void *pairs, int npairs, const int2 *queue, int nitems, void *scratch,
                          long long stride, int pitch, int rb, unsigned int *qhead, unsigned int *topq, int *status,
                          int *abort_flag, int blocks, cudaStream_t st, int keep_states, bool top_ef);
// theta > 0: the truncated base-match pass (min_am_prob = theta^2) after a
// full backward pass; theta = 0: the full adjoint pass, with the gap counts
// (the indel / indel-opening gradients) when grads
template <typename T>
cudaError_t pf_launch_back(const void *pairs, int npairs, const int2 *queue, int nitems, void *scratch,
                           long long stride, int pitch, int rb, unsigned int *qhead, unsigned int *topq, int *status,
                           int *abort_flag, int blocks, cudaStream_t st, double theta = 0.0, bool grads = true);
// w and D at the start of the forward pass; max_entries: most arc matches or band
// cells of a pair, dsw: offset of the structure weight
template <typename T>
cudaError_t pf_launch_entries(const void *pairs, const PFArcMatches *am, int npairs, int max_entries, double dsw,
                              double temperature, cudaStream_t st);
// PFArcMatches::prob, and bmacc over Z, after a backward pass
template <typename T>
cudaError_t pf_launch_probs(const void *pairs, const PFArcMatches *am, int npairs, int max_entries, cudaStream_t st);
// rb: ring size of the shared-memory rows (a power of two above the span of
// any two consecutive band rows)
template <typename T>
cudaError_t pf_fwd_occupancy(int rb, int *blocks_per_sm);
template <typename T>
cudaError_t pf_back_occupancy(int rb, int *blocks_per_sm);
int pf_warps_per_block();

cudaError_t pf_lane_occupancy(int rb, int *blocks_per_sm);
cudaError_t pf_launch_lane_fwd(const void *pairs, int npairs, const int2 *queue, int nitems, const PFLaneScratch &s, int rb,
                               unsigned int *qhead, unsigned int *topq, int *status, int *abort_flag, cudaStream_t st);
// theta as for pf_launch_back
cudaError_t pf_launch_lane_back(const void *pairs, int npairs, const int2 *queue, int nitems, const PFLaneScratch &s,
                                int rb, unsigned int *qhead, unsigned int *topq, int *status, int *abort_flag,
                                cudaStream_t st, double theta);

}  // namespace lcg
