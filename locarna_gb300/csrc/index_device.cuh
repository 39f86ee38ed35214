// Inputs and work arrays of the index kernels (index_kernels.cu), per pair
#pragma once
#include <cuda_runtime.h>

#include "lcg_device.cuh"

namespace lcg {

struct IndexPair {
    const int4 *arcs;  // per arc of A: l, r, first and past its last arc match (nullptr: the host made the index)
    const int *row_start, *row_arcs;  // arcs of A by right end
    const int4 *lefts;                // per left end of A: first and past its last arc, first and past its last group
    int nlefts;
    const int *am_lr;                 // per arc match: ends of its arc of B, l | r << 16
    const int *am_b, *inner_a, *inner_b;  // stacking: arc of B per arc match, next inner arc per arc (-1: none)
    const unsigned char *am_stackable;
    int *am_pos;            // per arc match its D index (-1: right ends outside the band)
    int *cursor, *gcursor;  // per band cell, per group
};

// pairs[q], ix[q] for q < npairs; max_n: longest A, max_lefts: most left ends
cudaError_t launch_index(const PairDev *pairs, const IndexPair *ix, int npairs, int max_n, int max_lefts,
                         cudaStream_t st);

}  // namespace lcg
