// Sequence envelope on the GPU: the trace-probability band of the reference's
// TraceController (trace_controller.cc:565-597) from the PFGotoh forward and
// reverse partition functions (edge_probs.icc:76-162) and the edge
// probabilities of PFTraceProbs (edge_probs.icc:212-268), for a batch of
// pairs, one block per pair (four warps per direction).
//
// 166 pairs of 60-400 nt take 5.0 ms and 0.3 ms for the weights; one warp per
// pair, four pairs per block, took 29.3 ms (FP64 issue of the 42 SMs it used),
// one warp per block with the weights kept for the reverse pass 18.3 ms (the
// row's chain of dependent FP64 operations).
//
// The reference evaluates the recursions in long double (locarna) or double
// (locarna_p) without scaling. Here every matrix row is kept in FP64 scaled by
// a power of two (exact), with its exponent alongside, so no row overflows.
// Only the threshold decision p(i,j) >= min_prob leaves the kernel: cells whose
// probability lies within a relative margin of the threshold (far above the
// FP64 and the reference's own rounding) are reported, and the host recomputes
// such a pair in the reference's precision when one of them could move a row
// bound. Pairs whose unscaled values would leave the range of the reference's
// float type are reported likewise (the reference's result there depends on
// its overflow behaviour).
//
// Matrices are full rows (n+1) x (m+1) as in the reference: out-of-band cells
// hold the values the reference leaves there (zero, or the free-end-gap and
// boundary initialisations of row 0 and column 0).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/locarna_gb300.h"
#include "engine_state.hh"
#include "envelope.hh"
#include "smem_limit.hh"

namespace {

constexpr int ENV_SIDE = 128;             // threads per direction
constexpr int ENV_THREADS = 2 * ENV_SIDE;  // forward and reverse pass of one pair
constexpr int ENV_ROW_SMEM = 96 * 1024;    // at most this much shared memory for rows, else they stay in HBM

struct EnvDev {
    int n, m;
    const signed char *ca, *cb;
    const double *sdA, *suA, *sdB, *suB;
    const int *minc, *maxc;
    int *newmin, *newmax, *flag;
    double *fz, *rz;    // forward and reverse rows: (n+1) x [zM | zA | zB] x (m+1)
    int *fexp, *rexp;   // their exponents
    double *wt;         // match weights, (n+1) x (m+1)
};

struct EnvConst {
    double sw, itemp, go, ge, gopen1, min_prob, mu;
    double score[16];
    int local, fe, rfe, exp_limit;
    int range;  // rows are scaled back once their largest value leaves 2^-range .. 2^range
};

// value = v * 2^e, v kept in [1, 2) (or 0)
struct XAcc {
    double v;
    int e;
};

__device__ __forceinline__ void xadd(XAcc &a, double v, int e) {
    if (v == 0.0) return;
    if (a.v == 0.0) {
        a.v = v;
        a.e = e;
    } else if (e > a.e) {
        a.v = ldexp(a.v, a.e - e) + v;
        a.e = e;
    } else {
        a.v += ldexp(v, e - a.e);
    }
    const int d = ilogb(a.v);
    a.v = ldexp(a.v, -d);
    a.e += d;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// band of row i in direction REV (the reverse band is TraceRange::reverse,
// trace_controller.cc:319-338)
template <bool REV>
__device__ __forceinline__ int band_lo(const EnvDev &P, int i) {
    return REV ? P.m - P.maxc[P.n - i] : P.minc[i];
}
template <bool REV>
__device__ __forceinline__ int band_hi(const EnvDev &P, int i) {
    return REV ? P.m - P.minc[P.n - i] : P.maxc[i];
}

// Boltzmann weight of the StralScore match (stral_score.cc:29-60) at (i, j).
// The reverse pass's object mirrors both sequences and swaps the up/down
// probabilities, which leaves sqrt(dA dB) + sqrt(uA uB) unchanged.
__device__ __forceinline__ double match_weight(const EnvDev &P, const EnvConst &C, int i, int j) {
    const int a = P.ca[i], b = P.cb[j];
    const double seq = (a >= 0 && b >= 0) ? C.score[a * 4 + b] : 0.0;
    const double s = C.sw * (P.sdA[i] * P.sdB[j] + P.suA[i] * P.suB[j]) + seq;
    return exp(s * C.itemp);
}

// The weights of every cell that a pass reads: cells of the band (forward) and
// those one step down and right of one (reverse). One warp per row; the exp
// evaluations are most of the envelope's FP64 operations, of which an SM issues
// two a clock, so they are spread over all SMs and done once for both passes.
__global__ void __launch_bounds__(256) env_weights_kernel(const EnvDev *__restrict__ pairs, EnvConst C) {
    const EnvDev &P = pairs[blockIdx.x];
    const int i = blockIdx.y * 8 + (threadIdx.x >> 5) + 1;
    if (i > P.n) return;
    const int lo = max(1, min(P.minc[i], P.minc[i - 1] + 1)), hi = min(P.m, max(P.maxc[i], P.maxc[i - 1] + 1));
    double *const w = P.wt + (size_t)i * (P.m + 1);
    for (int j = lo + (threadIdx.x & 31); j <= hi; j += 32) w[j] = match_weight(P, C, i, j);
}

// Constants of a warp's gap chains: g_ext^1, 2, 4, 8, 16 and g_ext^(lane+1)
struct EnvPow {
    double p[5], lane;
};
__device__ __forceinline__ EnvPow env_pow(double ge) {
    EnvPow w;
    double x = ge, y = ge;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        w.p[k] = x;
        if (lane >> k & 1) y *= x;
        x *= x;
    }
    w.lane = y;
    return w;
}

// what the four warps of a direction exchange
struct EnvShare {
    double a[2][4], t[2][4];  // gap-chain totals of a warp's 32 columns, by pass parity
    double sum[4], top[4];
    int hmax[4];
};


// One direction of the partition function (PFGotoh::pf_gotoh, edge_probs.icc:
// 76-162) by 128 threads: rows in order, 128 columns at a time. The gap chain
// of a row is a linear recurrence T(j) = a(j) T(j-1) + c(j): a scan inside each
// warp (constant factors where its 32 columns are all in the band), the warps'
// totals combined through shared memory. Rows are kept in HBM for the edge
// probabilities and, where they fit, two of them in shared memory. A row that
// has left 2^-range .. 2^range is scaled back to 1 .. 2 by a power of two
// (exact); zexp holds the exponents. Returns the flag (2: values that the
// reference's float type or the scaled FP64 rows would not hold); local alignment: *zloc, the sum of zM.
template <bool REV>
__device__ int env_pass(const EnvDev &P, const EnvConst &C, double *rows, EnvShare &sh, XAcc *zloc) {
    const int tid = threadIdx.x & (ENV_SIDE - 1), lane = tid & 31, sub = tid >> 5;
    const int n = P.n, m = P.m, m1 = m + 1;
    const size_t rowsz = 3 * (size_t)m1;
    double *const z = REV ? P.rz : P.fz;
    int *const zexp = REV ? P.rexp : P.fexp;
    const int fe = REV ? C.rfe : C.fe;
    const EnvPow W = env_pow(C.ge);
    const double gog = C.go * C.ge;
    auto sync = [] { asm volatile("bar.sync %0, %1;" ::"r"(REV ? 2 : 1), "n"(ENV_SIDE) : "memory"); };
    // row i's values: zM, zA, zB
    auto row = [&](int i) { return rows ? rows + (size_t)(i & 1) * rowsz : z + (size_t)i * rowsz; };
    int flag = 0, e = 0;
    {
        // row 0 (edge_probs.icc:89-117): zM(0,0) = 1 (global) / 0 (local);
        // zB(0,j) = g_open g_ext^j along the band; +1 on zB(0,j) with free end
        // gaps at the start of B
        double *const r = row(0);
        const int lo0 = band_lo<REV>(P, 0), hi0 = band_hi<REV>(P, 0);
        const bool chain = lo0 <= 1;
        for (int j = tid; j <= m; j += ENV_SIDE) {
            const double zm = (j == 0 && lo0 == 0 && !C.local) ? 1.0 : 0.0;
            double zb = 0.0;
            if (j >= 1) {
                if (chain && j <= hi0) zb = C.go * C.ge * pow(C.ge, (double)(j - 1));
                if (fe & LCG_FREE_LEFT_1) zb += 1.0;
            }
            r[j] = zm;
            r[m1 + j] = 0.0;
            r[2 * m1 + j] = zb;
            if (rows) {
                z[j] = zm;
                z[m1 + j] = 0.0;
                z[2 * m1 + j] = zb;
            }
        }
        if (tid == 0) zexp[0] = 0;
    }
    sync();
    for (int i = 1; i <= n; ++i) {
        const double *const prev = row(i - 1);
        double *const cur = row(i), *const out = z + (size_t)i * rowsz;
        const int lo = band_lo<REV>(P, i), hi = band_hi<REV>(P, i);
        const int j0 = max(lo, 1), j1 = min(hi, m);
        // column 0: zA(i,0) = g_open g_ext^i while the band holds column 0 (from
        // row 1 on), +1 with free end gaps at the start of A
        double col0 = 0.0;
        if (tid == 0) {
            if (band_lo<REV>(P, 1) == 0 && lo == 0) col0 = C.go * C.ge * pow(C.ge, (double)(i - 1));
            if (fe & LCG_FREE_LEFT_2) col0 += 1.0;
            col0 = ldexp(col0, -e);
        }
        const double locw = C.local ? ldexp(1.0, -e) : 0.0;
        const double *const w = P.wt + (size_t)(REV ? n + 1 - i : i) * m1;
        double carry = 0.0, rsum = 0.0;  // T of the column before the pass
        int hmax = 0, par = 0;
        for (int base = 0; base <= m; base += ENV_SIDE, par ^= 1) {
            const int j = base + tid;
            const bool act = j <= m, inb = act && j >= j0 && j <= j1;
            double zm = 0.0, za = col0;  // (zero but for column 0)
            col0 = 0.0;
            if (inb) {
                const double wj = w[REV ? m + 1 - j : j];
                const double pm1 = prev[j - 1] + prev[m1 + j - 1] + prev[2 * m1 + j - 1];
                zm = C.local ? pm1 * wj + wj * locw : pm1 * wj;
                za = prev[m1 + j] * C.ge + (prev[j] + prev[2 * m1 + j]) * gog;
            }
            // zB(j) = T(j-1) inside the band, 0 outside; T(j) = g_ext zB(j) + (zM + zA)(j) g_open g_ext
            double t = (zm + za) * gog, a;
            const int c0 = base + 32 * sub;
            if (c0 >= j0 && c0 + 31 <= j1) {
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const double t2 = __shfl_up_sync(0xffffffffu, t, 1 << k);
                    if (lane >= 1 << k) t = W.p[k] * t2 + t;
                }
                a = W.lane;
            } else {
                a = inb ? C.ge : 0.0;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const double a2 = __shfl_up_sync(0xffffffffu, a, off);
                    const double t2 = __shfl_up_sync(0xffffffffu, t, off);
                    if (lane >= off) {
                        t = a * t2 + t;
                        a = a * a2;
                    }
                }
            }
            if (lane == 31) {
                sh.a[par][sub] = a;
                sh.t[par][sub] = t;
            }
            sync();
            double c = carry;
            for (int s = 0; s < 4; ++s) {
                if (s == sub) c = carry;
                carry = sh.a[par][s] * carry + sh.t[par][s];
            }
            t = a * c + t;
            double zb = __shfl_up_sync(0xffffffffu, t, 1);
            if (lane == 0) zb = c;
            if (!inb) zb = 0.0;
            if (act) {
                cur[j] = zm;
                cur[m1 + j] = za;
                cur[2 * m1 + j] = zb;
                if (rows) {
                    out[j] = zm;
                    out[m1 + j] = za;
                    out[2 * m1 + j] = zb;
                }
                // no value is negative: their order is that of the high words
                hmax = max(hmax, max(__double2hiint(zm), max(__double2hiint(za), __double2hiint(zb))));
                if (C.local) rsum += zm;
            }
        }
        // the row's largest value and, local, its sum
        hmax = __reduce_max_sync(0xffffffffu, hmax);
        if (C.local) rsum = warp_sum(rsum);
        if (lane == 0) {
            sh.hmax[sub] = hmax;
            sh.sum[sub] = rsum;
        }
        sync();
        hmax = max(max(sh.hmax[0], sh.hmax[1]), max(sh.hmax[2], sh.hmax[3]));
        if (C.local && zloc) xadd(*zloc, sh.sum[0] + sh.sum[1] + sh.sum[2] + sh.sum[3], e);
        int d = (hmax >> 20) - 1023;
        if (hmax < 1 << 20) {  // zeros, or below the normal range
            double mx = 0.0;
            for (int k = tid; k < 3 * m1; k += ENV_SIDE) mx = fmax(mx, cur[k]);
            mx = warp_max(mx);
            if (lane == 0) sh.top[sub] = mx;
            sync();
            mx = fmax(fmax(sh.top[0], sh.top[1]), fmax(sh.top[2], sh.top[3]));
            d = mx > 0.0 ? ilogb(mx) : 0;
        }
        if (e + d + 2 > C.exp_limit || d > 1023) flag = 2;
        if (d > C.range || d < -C.range) {
            for (int k = tid; k < 3 * m1; k += ENV_SIDE) {
                const double v = ldexp(cur[k], -d);
                cur[k] = v;
                if (rows) out[k] = v;
            }
            e += d;
            sync();
        }
        if (tid == 0) zexp[i] = e;
    }
    return flag;
}

// One pair per block: forward and reverse pass side by side, then the edge
// probabilities (PFTraceProbs, edge_probs.icc:212-268) and row thresholds, a
// warp per row. Bound by FP64 issue and, for a pair alone, by the rows' chain of
// dependent FP64 operations (about 2,500 clocks a row of 400).
__global__ void __launch_bounds__(ENV_THREADS) envelope_kernel(const EnvDev *__restrict__ pairs, EnvConst C,
                                                               size_t row_smem) {
    extern __shared__ double env_smem[];
    __shared__ EnvShare share[2];
    __shared__ XAcc zloc_s;
    __shared__ int flags[3];
    const EnvDev &P = pairs[blockIdx.x];
    const int n = P.n, m = P.m, m1 = m + 1;
    const size_t rowsz = 3 * (size_t)m1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool rev = threadIdx.x >= ENV_SIDE;
    const bool shared_rows = 4 * rowsz * sizeof(double) <= row_smem;
    if (threadIdx.x == 0) flags[2] = 0;
    if (rev) {
        const int f = env_pass<true>(P, C, shared_rows ? env_smem + 2 * rowsz : nullptr, share[1], nullptr);
        if (threadIdx.x == ENV_SIDE) flags[1] = f;
    } else {
        XAcc zloc{0.0, 0};  // (zM of row 0 is 0 in local alignment)
        const int f = env_pass<false>(P, C, shared_rows ? env_smem : nullptr, share[0], &zloc);
        if (threadIdx.x == 0) {
            flags[0] = f;
            zloc_s = zloc;
        }
    }
    __syncthreads();
    // total (edge_probs.icc:220-236), every warp for itself
    const XAcc zloc = zloc_s;
    int flag = max(flags[0], flags[1]);
    XAcc z{0.0, 0};
    if (C.local) {
        xadd(z, 1.0, 0);
        xadd(z, zloc.v, zloc.e);
    } else {
        const double *rn = P.fz + (size_t)n * rowsz;
        const int e = P.fexp[n];
        xadd(z, rn[m] + rn[m1 + m] + rn[2 * m1 + m], e);
        if (C.fe & LCG_FREE_LEFT_2)
            for (int i = 0; i <= n; ++i) xadd(z, P.fz[(size_t)i * rowsz + m1 + m], P.fexp[i]);
        if (C.fe & LCG_FREE_LEFT_1) {
            double s = 0.0;
            for (int j = lane; j <= m; j += 32) s += rn[2 * m1 + j];
            xadd(z, warp_sum(s), e);
        }
    }
    if (z.v == 0.0 || z.e + 2 > C.exp_limit || z.e < -C.exp_limit) flag = 2;
    const double zinv = z.v > 0.0 ? 1.0 / z.v : 0.0;
    const double gopen_inv = 1.0 / C.gopen1;
    const double thr_hi = C.min_prob * (1.0 + C.mu), thr_lo = C.min_prob * (1.0 - C.mu);
    int unsure = 0;
    for (int i = warp; i <= n; i += ENV_THREADS / 32) {
        // edge probabilities of forward row i with reverse row n - i
        // (edge_probs.icc:238-262) and the row's threshold
        // (trace_controller.cc:568-579)
        const double *f = P.fz + (size_t)i * rowsz, *cur = P.rz + (size_t)(n - i) * rowsz;
        const int er = P.rexp[n - i], k = P.fexp[i] + er - z.e;
        const double locs = C.local ? ldexp(1.0, -er) : 0.0;
        const int lo = P.minc[i], hi = P.maxc[i];
        int nmin = hi, nmax = lo, umin = INT_MAX, umax = INT_MIN;
        // p = zij / z 2^k is compared as zij / z with the thresholds 2^-k, which
        // is exact while those stay in the normal range
        const bool direct = k > -900 && k < 900;
        const double t_hi = direct ? ldexp(thr_hi, -k) : thr_hi, t_lo = direct ? ldexp(thr_lo, -k) : thr_lo;
        for (int j = max(lo, 0) + lane; j <= min(hi, m); j += 32) {
            const int jr = m - j;
            const double rM = cur[jr], rA = cur[m1 + jr], rB = cur[2 * m1 + jr];
            const double zij = f[j] * (rM + rA + rB + locs) + f[m1 + j] * (rM + rA * gopen_inv + rB) +
                               f[2 * m1 + j] * (rM + rA + rB * gopen_inv);
            const double p = direct ? zij * zinv : ldexp(zij * zinv, k);
            if (p >= t_hi) {
                nmin = min(nmin, j);
                nmax = max(nmax, j);
            } else if (p >= t_lo) {
                umin = min(umin, j);
                umax = max(umax, j);
            }
        }
        nmin = __reduce_min_sync(0xffffffffu, nmin);
        nmax = __reduce_max_sync(0xffffffffu, nmax);
        umin = __reduce_min_sync(0xffffffffu, umin);
        umax = __reduce_max_sync(0xffffffffu, umax);
        if (umin < nmin || umax > nmax) unsure = 1;
        if (lane == 0) {
            P.newmin[i] = nmin;
            P.newmax[i] = nmax;
        }
    }
    if (lane == 0 && unsure) flags[2] = 1;  // (any writer writes the same)
    __syncthreads();
    if (threadIdx.x == 0) *P.flag = flag ? flag : flags[2];
}

size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

}  // namespace

namespace lcg_env {

void reset_transfer(lcg_engine eng) {
    eng->prep_h2d = 0;
    eng->prep_d2h = 0;
}

struct Pending {
    std::vector<std::pair<int, size_t>> outs;  // (pair, output offset in the pinned staging)
    PairOut *out = nullptr;
    const PairIn *in = nullptr;
    size_t out_begin = 0, out_end = 0;
    cudaEvent_t done = nullptr;
};

// One wave (pairs [q0, q1), wave_end) staged, enqueued and, with wait, finished;
// without wait the wave's outputs are described in *pend. LCG_ERR_NOMEM: nothing
// is enqueued.
static lcg_status enqueue_wave(lcg_engine eng, const EnvConst &C, int q0, int q1, const PairIn *in, PairOut *out,
                               bool wait, Pending *pend, std::string &err);

static EnvConst make_const(const Params &Pm, int npairs, const PairIn *in) {
    EnvConst C;
    C.sw = Pm.sw;
    C.itemp = 1.0 / Pm.temp;
    C.go = Pm.g_open;
    C.ge = Pm.g_ext;
    C.gopen1 = Pm.g_open;
    C.min_prob = Pm.min_prob;
    C.mu = 1e-7;  // relative margin around the threshold (FP64 rounding is below 1e-12 here)
    std::memcpy(C.score, Pm.score, sizeof C.score);
    C.local = Pm.local;
    C.fe = Pm.fe;
    int rfe = 0;  // FreeEndgaps::reverse (free_endgaps.hh:74-79)
    if (Pm.fe & LCG_FREE_LEFT_1) rfe |= LCG_FREE_RIGHT_1;
    if (Pm.fe & LCG_FREE_RIGHT_1) rfe |= LCG_FREE_LEFT_1;
    if (Pm.fe & LCG_FREE_LEFT_2) rfe |= LCG_FREE_RIGHT_2;
    if (Pm.fe & LCG_FREE_RIGHT_2) rfe |= LCG_FREE_LEFT_2;
    C.rfe = rfe;
    C.exp_limit = Pm.exp_limit;
    // A row may stay within 2^-128 .. 2^128 unscaled where a row's step (a match
    // weight, and a gap of any length) changes it by far less than the rest of
    // FP64's range; else every row is scaled to 1 .. 2, and the step has all of it.
    int max_m = 0;
    double score = 0.0;
    for (int q = 0; q < npairs; ++q) max_m = std::max(max_m, in[q].m);
    for (double s : Pm.score) score = std::max(score, std::fabs(s));
    const double step = (2.0 * std::fabs(Pm.sw) + score) * std::fabs(C.itemp) / std::log(2.0) +
                        std::fabs(std::log2(Pm.g_open)) + max_m * std::max(0.0, std::log2(Pm.g_ext));
    C.range = step < 256.0 ? 128 : 0;
    return C;
}

// device bytes of a pair beside its staged inputs: forward and reverse rows (three
// states each) and match weights, 56 bytes a cell, and the rows' exponents
static size_t pair_bytes(const PairIn &p) {
    const size_t n1 = (size_t)p.n + 1, m1 = (size_t)p.m + 1;
    return 8 * 7 * n1 * m1 + 8 * n1;
}

// the wave that starts with pair q0: at least that pair, and as many as the
// engine's budget takes
static int wave_end(lcg_engine eng, const PairIn *in, int q0, int npairs, size_t *bytes = nullptr) {
    size_t sum = pair_bytes(in[q0]);
    int q1 = q0 + 1;
    for (; q1 < npairs && sum + pair_bytes(in[q1]) <= eng->env_wave_bytes; ++q1) sum += pair_bytes(in[q1]);
    if (bytes) *bytes = sum;
    return q1;
}

lcg_status compute(lcg_engine eng, const Params &Pm, int npairs, const PairIn *in, PairOut *out, std::string &err) {
    if (npairs <= 0) return LCG_OK;
    cudaError_t ce = cudaSetDevice(eng->device);
    if (ce != cudaSuccess) {
        err = std::string("cudaSetDevice: ") + cudaGetErrorString(ce);
        return LCG_ERR_CUDA;
    }
    const EnvConst C = make_const(Pm, npairs, in);
    for (int q0 = 0; q0 < npairs;) {
        size_t bytes;
        const int q1 = wave_end(eng, in, q0, npairs, &bytes);
        const lcg_status rc = enqueue_wave(eng, C, q0, q1, in, out, true, nullptr, err);
        if (rc == LCG_ERR_NOMEM && q1 - q0 > 1) {
            eng->env_wave_bytes = bytes / 2;  // in smaller waves
            continue;
        }
        if (rc == LCG_ERR_NOMEM) out[q0].flag = 2;  // a pair too large for the memory left: the host's
        else if (rc != LCG_OK) return rc;
        q0 = q1;
    }
    return LCG_OK;
}

lcg_status compute_begin(lcg_engine eng, const Params &Pm, int npairs, const PairIn *in, PairOut *out,
                         Pending **pending, std::string &err) {
    *pending = nullptr;
    if (npairs <= 0) return LCG_OK;
    cudaError_t ce = cudaSetDevice(eng->device);
    if (ce != cudaSuccess) {
        err = std::string("cudaSetDevice: ") + cudaGetErrorString(ce);
        return LCG_ERR_CUDA;
    }
    // more than one wave: computed now (the pinned staging holds one wave)
    size_t bytes;
    if (wave_end(eng, in, 0, npairs, &bytes) < npairs) return compute(eng, Pm, npairs, in, out, err);
    auto *p = new Pending;
    lcg_status rc = enqueue_wave(eng, make_const(Pm, npairs, in), 0, npairs, in, out, false, p, err);
    if (rc != LCG_OK) {
        if (p->done) cudaEventDestroy(p->done);
        delete p;
        if (rc != LCG_ERR_NOMEM) return rc;
        eng->env_wave_bytes = bytes / 2;
        return compute(eng, Pm, npairs, in, out, err);
    }
    *pending = p;
    return LCG_OK;
}

lcg_status compute_end(lcg_engine eng, Pending *p, std::string &err) {
    if (!p) return LCG_OK;
    const cudaError_t ce = cudaEventSynchronize(p->done);
    cudaEventDestroy(p->done);
    if (ce != cudaSuccess) {
        err = std::string("envelope kernel: ") + cudaGetErrorString(ce);
        delete p;
        return LCG_ERR_CUDA;
    }
    const char *H = eng->env_host;
    eng->prep_h2d += (long long)p->out_begin;
    eng->prep_d2h += (long long)(p->out_end - p->out_begin);
    for (auto &x : p->outs) {
        const int n1 = p->in[x.first].n + 1;
        const int *o = (const int *)(H + x.second);
        std::memcpy(p->out[x.first].newmin, o, 4ull * n1);
        std::memcpy(p->out[x.first].newmax, o + n1, 4ull * n1);
        p->out[x.first].flag = o[2 * n1];
    }
    delete p;
    return LCG_OK;
}

static lcg_status enqueue_wave(lcg_engine eng, const EnvConst &C, int q0, int q1, const PairIn *in, PairOut *out,
                               bool wait, Pending *pend, std::string &err) {
    cudaError_t ce;
    std::vector<size_t> in_off, out_off, dev_off;
    auto take = [](size_t &cur, size_t b) {
        size_t o = cur;
        cur = align16(cur + b);
        return o;
    };
    const int nq = q1 - q0;
    // host staging: [EnvDev x nq][per pair inputs][per pair outputs]
    size_t hs = 0;
    const size_t o_pairs = take(hs, sizeof(EnvDev) * nq);
    in_off.resize(nq);
    for (int k = 0; k < nq; ++k) {
        const PairIn &p = in[q0 + k];
        const size_t n1 = (size_t)p.n + 1, m1 = (size_t)p.m + 1;
        in_off[k] = take(hs, 4 * (2 * n1) + 8 * (2 * n1 + 2 * m1) + n1 + m1);
    }
    const size_t out_begin = hs;
    out_off.resize(nq);
    for (int k = 0; k < nq; ++k) out_off[k] = take(hs, 4 * (2 * ((size_t)in[q0 + k].n + 1) + 1));
    const size_t out_end = hs;
    size_t ds = hs;  // device-only section after the mirrored staging
    dev_off.resize(nq);
    for (int k = 0; k < nq; ++k) dev_off[k] = take(ds, pair_bytes(in[q0 + k]));
    // the buffers are reused only after the previous computation ended
    // (compute waits; a pending one is ended before the next begins)
    if (ds > eng->env_dev_cap) {
        if (eng->env_dev) cudaFree(eng->env_dev);
        eng->env_dev = nullptr;
        eng->env_dev_cap = 0;
        // with room to grow, else without; else the caller takes a smaller wave
        for (size_t cap : {ds + std::min<size_t>(ds / 4, (size_t)1 << 30), ds})
            if (!eng->env_dev_cap && lcg_host::device_alloc(&eng->env_dev, cap) == cudaSuccess) eng->env_dev_cap = cap;
        if (!eng->env_dev_cap) {
            err = "envelope device allocation failed";
            return LCG_ERR_NOMEM;
        }
    }
    if (out_end > eng->env_host_cap) {
        if (eng->env_host) cudaFreeHost(eng->env_host);
        eng->env_host = nullptr;
        eng->env_host_cap = 0;
        if (cudaMallocHost(&eng->env_host, out_end + out_end / 4) != cudaSuccess) {
            cudaGetLastError();
            eng->env_host = nullptr;
            err = "envelope pinned allocation failed";
            return LCG_ERR_NOMEM;
        }
        eng->env_host_cap = out_end + out_end / 4;
    }
    char *H = eng->env_host, *D = eng->env_dev;
    EnvDev *hp = (EnvDev *)(H + o_pairs);
    // the largest pairs first: they take longest, and blocks start in this order
    std::vector<int> order(nq);
    for (int k = 0; k < nq; ++k) order[k] = k;
    auto area = [&](int k) { return (long long)in[q0 + k].n * in[q0 + k].m; };
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return area(x) > area(y); });
    for (int r = 0; r < nq; ++r) {
        const int k = order[r];
        const PairIn &p = in[q0 + k];
        const int n1 = p.n + 1, m1 = p.m + 1;
        char *h = H + in_off[k];
        char *d = D + in_off[k];
        int *minc = (int *)h, *maxc = minc + n1;
        std::memcpy(minc, p.minc, 4ull * n1);
        std::memcpy(maxc, p.maxc, 4ull * n1);
        double *sdA = (double *)(h + 8ull * n1), *suA = sdA + n1, *sdB = suA + n1, *suB = sdB + m1;
        std::memcpy(sdA, p.sdA, 8ull * n1);
        std::memcpy(suA, p.suA, 8ull * n1);
        std::memcpy(sdB, p.sdB, 8ull * m1);
        std::memcpy(suB, p.suB, 8ull * m1);
        signed char *ca = (signed char *)(suB + m1), *cb = ca + n1;
        std::memcpy(ca, p.ca, n1);
        std::memcpy(cb, p.cb, m1);
        EnvDev &v = hp[r];
        v.n = p.n;
        v.m = p.m;
        v.minc = (const int *)d;
        v.maxc = (const int *)d + n1;
        v.sdA = (const double *)(d + 8ull * n1);
        v.suA = v.sdA + n1;
        v.sdB = v.suA + n1;
        v.suB = v.sdB + m1;
        v.ca = (const signed char *)(v.suB + m1);
        v.cb = v.ca + n1;
        char *od = D + out_off[k];
        v.newmin = (int *)od;
        v.newmax = (int *)od + n1;
        v.flag = (int *)od + 2 * n1;
        char *dd = D + dev_off[k];
        v.fz = (double *)dd;
        v.rz = v.fz + 3ull * n1 * m1;
        v.wt = v.rz + 3ull * n1 * m1;
        v.fexp = (int *)(v.wt + (size_t)n1 * m1);
        v.rexp = v.fexp + n1;
    }
    cudaStream_t st = eng->stream;
    auto fail_cuda = [&](cudaError_t x, const char *what) {
        err = std::string(what) + ": " + cudaGetErrorString(x);
        cudaStreamSynchronize(st);
        return LCG_ERR_CUDA;
    };
    if ((ce = cudaMemcpyAsync(D, H, out_begin, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return fail_cuda(ce, "envelope upload");
    int max_n = 1, max_m = 1;
    for (int k = 0; k < nq; ++k) {
        max_n = std::max(max_n, in[q0 + k].n);
        max_m = std::max(max_m, in[q0 + k].m);
    }
    env_weights_kernel<<<dim3(nq, (max_n + 7) / 8), 256, 0, st>>>((const EnvDev *)(D + o_pairs), C);
    const size_t smem = std::min<size_t>(ENV_ROW_SMEM, 4 * 3 * sizeof(double) * (size_t)(max_m + 1));
    if ((ce = lcg::allow_smem((const void *)envelope_kernel, smem)) != cudaSuccess)
        return fail_cuda(ce, "envelope launch");
    envelope_kernel<<<nq, ENV_THREADS, smem, st>>>((const EnvDev *)(D + o_pairs), C, smem);
    if ((ce = cudaGetLastError()) != cudaSuccess) return fail_cuda(ce, "envelope launch");
    if ((ce = cudaMemcpyAsync(H + out_begin, D + out_begin, out_end - out_begin, cudaMemcpyDeviceToHost, st)) !=
        cudaSuccess)
        return fail_cuda(ce, "envelope download");
    if (!wait) {
        // finished by compute_end: an event after the download
        if ((ce = cudaEventCreateWithFlags(&pend->done, cudaEventDisableTiming)) != cudaSuccess)
            return fail_cuda(ce, "envelope event");
        if ((ce = cudaEventRecord(pend->done, st)) != cudaSuccess) return fail_cuda(ce, "envelope event");
        pend->in = in;
        pend->out = out;
        pend->out_begin = out_begin;
        pend->out_end = out_end;
        for (int k = 0; k < nq; ++k) pend->outs.emplace_back(q0 + k, out_off[k]);
        return LCG_OK;
    }
    if ((ce = cudaStreamSynchronize(st)) != cudaSuccess) return fail_cuda(ce, "envelope kernel");
    eng->prep_h2d += (long long)out_begin;
    eng->prep_d2h += (long long)(out_end - out_begin);
    for (int k = 0; k < nq; ++k) {
        const int n1 = in[q0 + k].n + 1;
        const int *o = (const int *)(H + out_off[k]);
        std::memcpy(out[q0 + k].newmin, o, 4ull * n1);
        std::memcpy(out[q0 + k].newmax, o + n1, 4ull * n1);
        out[q0 + k].flag = o[2 * n1];
    }
    return LCG_OK;
}

}  // namespace lcg_env
