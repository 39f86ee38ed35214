// Device routines shared by the LocARNA-P kernels (pf_kernels.cu, which has the
// recursions, and pf_lane_kernels.cu): waits, the rows in shared memory, and the
// top level's sweeps.
#pragma once
#include <cuda_runtime.h>

#include <climits>

#include "lcg_device.cuh"
#include "pf_device.cuh"

namespace lcg {

constexpr int PF_WARPS = 4;
// resident blocks per SM the register budget targets: 8 (32 warps) in FP32;
// FP64 rows take twice the shared memory, 5 blocks fit
template <typename T>
__host__ __device__ constexpr int pf_min_blocks() {
    return sizeof(T) == 4 ? 8 : 5;
}
constexpr long long PF_SPIN_LIMIT = 1ll << 22;

__device__ __forceinline__ bool pf_not_ready(double v) {
    return __double_as_longlong(v) == PF_NOT_READY_F64;
}
__device__ __forceinline__ bool pf_not_ready(float v) { return __float_as_int(v) == PF_NOT_READY_F32; }
__device__ __forceinline__ double pf_ld(const double *p) { return *(const volatile double *)p; }
__device__ __forceinline__ float pf_ld(const float *p) { return *(const volatile float *)p; }

template <typename T>
__device__ __forceinline__ T pf_wait(const T *p, int *status, volatile int *abort_flag) {
    T v = pf_ld(p);
    long long spins = 0;
    while (pf_not_ready(v)) {
        __nanosleep(64);
        v = pf_ld(p);
        if (++spins > PF_SPIN_LIMIT || *abort_flag) {
            atomicOr(status, ST_TIMEOUT);
            *abort_flag = 1;
            return T(0);
        }
    }
    return v;
}

// The gap chains' factors of a pair whose columns all have the same gap weight
// g (single sequences): g^1, 2, 4, 8, 16 for the warp scans (the carries take
// gpow[lane + 1] and gpow[32 - lane]). FP64 arithmetic is what bounds the FP64
// passes (an SM issues two FP64 operations a clock), and the scan with constant
// factors takes 5 multiply-adds a cell instead of 10. The powers come rounded
// once from the host: squared up here, g^16 was up to 15 roundings off, which the
// sweeps of lanes and of rows did not share (80 against 439 nt in FP32: am_prob
// 2.2e-6 off in norm).
template <typename T>
struct PFPow {
    T p[5];
};
// With gap gradients the FP32 sweeps keep the scan of pairs (a, b), and gu is then 0
// in all of them, so that all round a run of gaps alike: at 64 registers the factors
// cost that backward pass more than they save (28 pairs of 160-200 nt: 26.5 ms
// against 25.7; without gap gradients a 200-nt pair 2.43 ms against 2.64).
template <typename T>
__host__ __device__ constexpr bool pf_factors(bool grads) {
    return sizeof(T) == 8 || !grads;
}
template <typename T>
__device__ __forceinline__ PFPow<T> pf_pow(const PFPair<T> &P) {
    PFPow<T> w;
#pragma unroll
    for (int k = 0; k < 5; ++k) w.p[k] = P.gpow[1 << k];
    return w;
}

extern __shared__ unsigned char pf_smem_raw[];

// Shared-memory rows per warp (T each), ring buffers of rb entries (a
// multiple of 32) indexed by column j mod rb: M and N of the previous / current row, E, and
// the arc-term sums of the current row. RB exceeds the span of any two
// consecutive band rows, so live columns never alias. The backward pass
// reuses E as E_bar and Ar as the row's X_bar.
template <typename T>
struct PFRows {
    T *Mp, *Mc, *Np, *Nc, *E, *Ar;
    int rb;
    unsigned magic;  // j / rb = umulhi(j, magic) for 0 <= j < 2^20
};

constexpr int PF_RING_ROWS = 6;

template <typename T>
__device__ __forceinline__ PFRows<T> pf_rows(int warp, int rb) {
    T *base = reinterpret_cast<T *>(pf_smem_raw) + (size_t)warp * PF_RING_ROWS * rb;
    PFRows<T> r;
    r.Mp = base;
    r.Mc = base + rb;
    r.Np = base + 2 * rb;
    r.Nc = base + 3 * rb;
    r.E = base + 4 * rb;
    r.Ar = base + 5 * rb;
    r.rb = rb;
    r.magic = 0xFFFFFFFFu / (unsigned)rb + 1u;
    return r;
}

template <typename T>
__device__ __forceinline__ T ld_cg(const T *p) { return __ldcg(p); }

// ---- top levels: a whole block per pair
//
// A pair's top level is the last to finish in the forward pass and the first to
// go in the backward, where every group waits for it; it is the widest sweep
// and has the longest entry lists. By one warp a row of a 200-nt pair took 6.5 us
// forward and 13 us backward, 4.0 of the backward's 4.7 ms. A block spreads the
// row's columns and entries over its threads, and the backward reads what the
// forward kept: backward 4.7 -> 3.6 ms (top level 4.0 -> 1.6), forward 2.1 -> 1.9
// (the top level now after the groups, 1.2 ms); the truncated pass over ten pairs
// of 80-240 nt, which is little else, 2.1 -> 0.9. A row costs 6 to 8 us still:
// some 20 FP64 operations a column at 2 a clock per SM, L2 latency of M_bar and
// of the entries, and the fence before the counters. Entries
// loaded a row ahead, two columns a thread and longer naps of the waiting warps
// changed nothing.

// The recurrence x -> a x + b over the block's threads, in thread order, from
// the value c before the first one (the same in all threads): c becomes the
// value after the last thread, the result is the value before this thread and
// *own the one after it. W: the powers of a where all threads have the same a
// (then pa = a^(lane + 1)), else nullptr. sm: 2 PF_WARPS values, not the ones of
// the last call.
template <typename T>
__device__ __forceinline__ T pf_block_scan(T a, T b, const PFPow<T> *W, T pa, T &c, T *own, T *sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (W) {
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const T b1 = __shfl_up_sync(0xffffffffu, b, 1 << k);
            if (lane >= 1 << k) b += W->p[k] * b1;
        }
        a = pa;
    } else {
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const T a1 = __shfl_up_sync(0xffffffffu, a, off);
            const T b1 = __shfl_up_sync(0xffffffffu, b, off);
            if (lane >= off) {
                b = a * b1 + b;
                a = a * a1;
            }
        }
    }
    if (lane == 31) {
        sm[2 * warp] = a;
        sm[2 * warp + 1] = b;
    }
    __syncthreads();
    T before = c;
#pragma unroll
    for (int w = 0; w < PF_WARPS; ++w) {
        if (w == warp) before = c;
        c = sm[2 * w] * c + sm[2 * w + 1];
    }
    *own = a * before + b;
    const T left = __shfl_up_sync(0xffffffffu, *own, 1);
    return lane == 0 ? before : left;
}

// The forward sweep of a pair's top level (pf_group_sweep<SAVE> over all rows
// and columns) by a block: M to P.topM, with EF also E and F to Eg and Fg.
template <typename T, bool WAIT, bool COUNTU, bool EF>
__device__ __noinline__ void pf_top_sweep(const PFPair<T> &P, T *__restrict__ Eg, T *__restrict__ Fg, PFRows<T> R, T (*sm)[2 * PF_WARPS],
                             int *status, volatile int *abort_flag) {
    const int tid = threadIdx.x;
    constexpr int NT = PF_WARPS * 32;
    const int n = P.n, m = P.m, pitch = m + 1;
    const T o = P.o, arcf = P.arcf;
    T *const Mg = P.topM;
    const bool uni = P.gu > T(0);
    const PFPow<T> W = pf_pow(P);
    const T pa = P.gpow[(tid & 31) + 1];
#define RG(j) ((j) - R.rb * (int)__umulhi((unsigned)(j), R.magic))
    for (int c = tid; c < R.rb; c += NT) R.E[c] = R.Ar[c] = T(0);
    auto put = [&](size_t at, T M, T E, T F) {
        Mg[at] = M;
        if (EF) {
            Eg[at] = E;
            Fg[at] = F;
        }
    };
    int bf = 0;
    {
        // row 0: M(0,0) = 1/s, M(0,j) = (o/s) prod gB
        const int L0 = P.rowinfo[0].y + 1;
        T c = o * P.inv_s;
        for (int base = 1; base < L0; base += NT, bf ^= 1) {
            const int j = base + tid;
            T v;
            pf_block_scan<T>(j < L0 ? P.gB[j] : T(1), T(0), uni ? &W : nullptr, pa, c, &v, sm[bf]);
            if (j < L0) {
                R.Mp[RG(j)] = R.Np[RG(j)] = v;
                put(j, v, T(0), T(0));
            }
        }
        if (tid == 0) {
            R.Mp[0] = R.Np[0] = P.inv_s;
            put(0, P.inv_s, T(0), T(0));
        }
        for (int j = L0 + tid; j <= P.rowinfo[1].y; j += NT) {
            R.Mp[RG(j)] = R.Np[RG(j)] = T(0);
            put(j, T(0), T(0), T(0));
        }
    }
    T colval = o * P.inv_s;
    for (int i = 1; i <= n; ++i) {
        __syncthreads();  // the row above, its entry sums cleared
        const int4 ri = P.rowinfo[i];
        const int2 ra = P.rowarc[i];
        const int lo = max(1, ri.x), hi = ri.y;
        const T gAi = P.gA[i], gAo = gAi * o;
        const size_t row = (size_t)i * pitch;
        for (int e = ra.x + tid; e < ra.y; e += NT) {
            const int2 en = P.crow[e];
            if (en.y < lo || en.y > hi) continue;
            T dv = pf_ld(P.D + e);
            const T mv = Mg[(size_t)(en.x & 0xffff) * pitch + (en.x >> 16)];
            if (WAIT && pf_not_ready(dv)) dv = pf_wait(P.D + e, status, abort_flag);
            atomicAdd(&R.Ar[RG(en.y)], mv * dv);
            if (COUNTU) atomicAdd(P.cnt + e, 1);
        }
        T B = T(0);
        if (ri.x <= 0) B = colval *= gAi;
        if (tid == 0) {
            R.Mc[RG(lo - 1)] = R.Nc[RG(lo - 1)] = B;
            put(row + lo - 1, B, T(0), T(0));
        }
        __syncthreads();
        // F(j+1) = gB(j+1) (F(j) + o Q(j)): the value before thread j is F(j)
        T Fc = P.gB[min(lo, m)] * o * B;
        for (int base = lo; base <= hi; base += NT, bf ^= 1) {
            const int j = base + tid;
            const bool act = j <= hi;
            T X = T(0), Ei = T(0), a = T(1), b = T(0), own;
            if (act) {
                Ei = R.E[RG(j)] * gAi + R.Np[RG(j)] * gAo;
                X = R.Mp[RG(j - 1)] * P.bm[row + j];
                if (ra.x < ra.y) {
                    X += R.Ar[RG(j)] * arcf;
                    R.Ar[RG(j)] = T(0);
                }
                a = uni ? P.gu : j < m ? P.gB[j + 1] : T(0);
                b = a * o * (X + Ei);
            }
            const T F = pf_block_scan<T>(a, b, uni ? &W : nullptr, pa, Fc, &own, sm[bf]);
            if (act) {
                const T N = X + F, M = N + Ei;
                R.E[RG(j)] = Ei;
                R.Mc[RG(j)] = M;
                R.Nc[RG(j)] = N;
                put(row + j, M, Ei, F);
            }
        }
        if (i < n)
            // columns entering the band with row i+1 start from zero
            for (int j = max(hi + 1, 1) + tid; j <= P.rowinfo[i + 1].y; j += NT) {
                R.Mc[RG(j)] = R.Nc[RG(j)] = R.E[RG(j)] = T(0);
                put(row + j, T(0), T(0), T(0));
            }
        T *t;
        t = R.Mp; R.Mp = R.Mc; R.Mc = t;
        t = R.Np; R.Np = R.Nc; R.Nc = t;
    }
    __syncthreads();
#undef RG
}

// the next pair whose top level this block takes (npairs: none left)
__device__ __forceinline__ int pf_next_top(unsigned int *topq, int npairs, volatile int *abort_flag) {
    __shared__ int next;
    __syncthreads();
    if (threadIdx.x == 0) next = *abort_flag ? npairs : min((int)atomicAdd(topq, 1u), npairs);
    __syncthreads();
    return next;
}

// pf_group_back of a pair's top level, by a block: dZ'/dM(n,m) = 1 is the
// seed, all entries of a row are inside, and the row's columns go to the threads
// from right to left. Mg, Eg, Fg as pf_top_sweep wrote them.
template <typename T, bool TRUNC, bool GRADS>
__device__ __noinline__ void pf_top_back(const PFPair<T> &P, const T *__restrict__ Mg, const T *__restrict__ Eg,
                            const T *__restrict__ Fg, T *__restrict__ Mb, PFRows<T> R, T (*sm)[2 * PF_WARPS],
                            double *ext_acc, double *open_acc) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NT = PF_WARPS * 32;
    const int n = P.n, m = P.m, pitch = m + 1;
    const T o = P.o, arcf = P.arcf;
    T *const Eb = R.E, *const Xb = R.Ar;
    T *Dn = R.Mp, *Dc = R.Mc;  // diagonal contributions, as in pf_group_back
    const bool uni = P.gu > T(0);
    const PFPow<T> W = pf_pow(P);
    const T pa = P.gpow[lane + 1];
#define RG(j) ((j) - R.rb * (int)__umulhi((unsigned)(j), R.magic))
    for (int i = warp; i <= n; i += PF_WARPS) {
        const int hi = max(P.rowinfo[i].y, i < n ? P.rowinfo[i + 1].y : 0);
        for (int j = max(0, P.rowinfo[i].x - 1) + lane; j <= hi; j += 32) Mb[(size_t)i * pitch + j] = T(0);
        if (lane == 0) Mb[(size_t)i * pitch] = T(0);
    }
    for (int c = tid; c < R.rb; c += NT) Eb[c] = Dn[c] = Dc[c] = T(0);
    __syncthreads();
    if (tid == 0) Mb[(size_t)n * pitch + m] = T(1);
    double ext = 0.0, opn = 0.0;
    int bf = 0;
    for (int i = n; i > 0; --i) {
        __syncthreads();  // M_bar and the rings as row i+1 left them
        const int4 ri = P.rowinfo[i], rup = P.rowinfo[i - 1];
        const int2 ra = P.rowarc[i];
        const int lo = max(1, ri.x), hi = ri.y;
        const T gAi = P.gA[i], gAn = i < n ? P.gA[i + 1] : T(0);
        const T gAo = gAi * o, gAno = gAn * o;
        const size_t row = (size_t)i * pitch;
        const int cb = ri.w - ri.x;
        const int dlo = i > 1 ? max(1, rup.x) : INT_MAX, dhi = rup.y;
        // the thread's first entry, loaded ahead of the cells
        const int e0 = ra.x + tid;
        int2 en = make_int2(0, 0);
        T dv = T(0), mv = T(0);
        if (e0 < ra.y) {
            en = P.crow[e0];
            dv = P.D[e0];
            mv = Mg[(size_t)(en.x & 0xffff) * pitch + (en.x >> 16)];
        }
        T Fbc = T(0);
        T opnE = T(0);  // GRADS in FP64: the row's vertical gap openings without their weight
        for (int top = hi; top >= lo; top -= NT, bf ^= 1) {
            const int j = top - tid;
            const bool act = j >= lo;
            const size_t c = row + j;
            T Mbar = T(0), Ebn = T(0), gn = T(0), bmj = T(0), Md = T(0), own;
            if (act) {
                Mbar = ld_cg(Mb + c) + Dc[RG(j)];
                Dc[RG(j)] = T(0);
                Ebn = Eb[RG(j)];
                gn = uni ? P.gu : j < hi ? P.gB[j + 1] : T(0);
                bmj = P.bm[c];
                Md = Mg[c - pitch - 1];
            }
            const T MN = Mbar + Ebn * gAno;
            // F_bar(j) = gB(j+1) F_bar(j+1) + (M_bar + N_bar)(j)
            const T Fbr = pf_block_scan<T>(act ? gn : T(1), MN, uni ? &W : nullptr, pa, Fbc, &own, sm[bf]);
            const T Fb = own;
            if (act) {
                const T Qbar = Fbr * gn * o;
                const T Ebar = Mbar + (Qbar + Ebn * gAn);
                const T Xbar = MN + Qbar;
                Eb[RG(j)] = Ebar;
                Xb[RG(j)] = Xbar;
                if (GRADS) {
                    ext += (double)(Ebar * Eg[c] + Fb * Fg[c]);
                    const T down = Ebar * (Mg[c - pitch] - Eg[c - pitch]);
                    const T right = Fb * (Mg[c - 1] - Fg[c - 1]) * (P.gB[j] * o);
                    if (sizeof(T) == 8) {
                        opnE += down;
                        opn += (double)right;
                    } else {
                        opn += (double)(down * gAo + right);
                    }
                }
                const T Xd = Xbar * bmj;
                if (j - 1 >= dlo && j - 1 <= dhi)
                    Dn[RG(j - 1)] = Xd;
                else
                    atomicAdd(Mb + c - pitch - 1, Xd);
                atomicAdd(P.bmacc + cb + j, (double)(Xd * Md));
                if (i == 1 || rup.x > j || rup.y < j) atomicAdd(Mb + c - pitch, Ebar * gAo);
                if (j == lo) atomicAdd(Mb + c - 1, Fb * (P.gB[j] * o));
            }
        }
        if (GRADS && sizeof(T) == 8) opn += (double)opnE * gAo;
        __syncthreads();
        for (int e = e0; e < ra.y; e += NT) {
            if (e != e0) {
                en = P.crow[e];
                dv = P.D[e];
                mv = Mg[(size_t)(en.x & 0xffff) * pitch + (en.x >> 16)];
            }
            if (en.y < lo || en.y > hi) continue;
            const T xs = Xb[RG(en.y)] * arcf;
            atomicAdd(Mb + (size_t)(en.x & 0xffff) * pitch + (en.x >> 16), xs * dv);
            if (!TRUNC) atomicAdd(P.Dbar + e, (double)(xs * mv));
        }
        if (!TRUNC && e0 < ra.y) {
            __threadfence();  // the D_bar updates are visible before the counters drop
            for (int e = e0; e < ra.y; e += NT) {
                const int j = e == e0 && ra.y - e0 <= NT ? en.y : P.crow[e].y;
                if (j >= lo && j <= hi) atomicSub(P.cnt + e, 1);
            }
        }
        // E_bar of row i at columns row i-1 has but row i does not is zero
        if (i > 1)
            for (int j = max(1, rup.x) + tid; j < lo; j += NT) Eb[RG(j)] = T(0);
        T *const dt = Dn;
        Dn = Dc;
        Dc = dt;
    }
    __syncthreads();
#undef RG
    if constexpr (GRADS && !TRUNC) {
        for (int j = 1 + tid; j <= P.rowinfo[0].y; j += NT) {
            const T v = ld_cg(Mb + j) * Mg[j];
            ext += (double)v * j;
            opn += (double)v;
        }
        for (int i = 1 + tid; i <= n; i += NT) {
            if (P.rowinfo[i].x > 0) continue;
            const T v = ld_cg(Mb + (size_t)i * pitch) * Mg[(size_t)i * pitch];
            ext += (double)v * i;
            opn += (double)v;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            ext += __shfl_xor_sync(0xffffffffu, ext, off);
            opn += __shfl_xor_sync(0xffffffffu, opn, off);
        }
        if (lane == 0) {
            atomicAdd(ext_acc, ext);
            atomicAdd(open_acc, opn);
        }
    }
}

}  // namespace lcg
