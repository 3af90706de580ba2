// weights.cuh -- WeightSet updates and prospective ESS / CESS on device
// arrays (core/weight_set.hpp:108-186, 297-331, 385-431).
//
// The sums are online log-sum-exp accumulators (m, s1 = sum exp(l - m),
// s2 = sum exp(2 (l - m))) in one fixed association: 8 strided elements per
// thread in order, a shuffle tree, the 8 warps in order; then the tiles,
// contiguous runs per thread of 1024, a shuffle tree, the 32 warps in order.
// Of the two exponentials a step of the accumulator has, one is always
// exp(0) = 1: each step evaluates the other only, and a thread's 8 elements
// evaluate theirs independently of each other (the running maxima come
// first).  Loads are issued before the first store, so they overlap.
//
// Up to kWcTiles tiles (65536 elements) one cluster does the whole call in
// one launch, the log-weights staying in registers between the sums and the
// normalisation; larger arrays take sums, join and normalisation kernels.
// Bound: latency of launches and of the ordered joins below about 10^6
// elements, HBM / L2 above.  Measured on one B200 (a program's whole step of
// ESS, CESS, update, resampling and gather, most of the gain that of
// call_scratch.hpp's allocations): 1000 particles 1620 -> 102 us, 3000001
// particles 1950 -> 343 us.
#pragma once

#include <cooperative_groups.h>

#include "smc_common.cuh"

namespace vsmc_b200 {

struct WeightCtl {
    double M, S1, S2;
    int error;
};

struct WAcc {
    double m, s1, s2;

    __device__ __forceinline__ void init(double ref)
    {
        m = ref;
        s1 = s2 = 0.0;
    }

    // exp of a difference <= 0 that is 1 without evaluation when it is 0
    // (NaN for infinite references, as inf - inf gives)
    __device__ static __forceinline__ double one(double ref)
    {
        return ref < INFINITY ? 1.0 : NAN;
    }

    __device__ __forceinline__ void merge(const WAcc &o)
    {
        if (o.m == -INFINITY && o.s1 == 0.0)
            return;
        const double nm = fmax(m, o.m);
        const double x = exp(fmin(m, o.m) - nm);
        const double fa =
            m == -INFINITY ? 0.0 : (m == nm ? one(nm) : x);
        const double fb =
            o.m == -INFINITY ? 0.0 : (o.m == nm ? one(nm) : x);
        s1 = __fma_rn(s1, fa, __dmul_rn(o.s1, fb));
        s2 = __fma_rn(__dmul_rn(s2, fa), fa,
                      __dmul_rn(__dmul_rn(o.s2, fb), fb));
        m = nm;
    }
};

// The 8 log-weights of a thread into its accumulator, in order.
__device__ __forceinline__ void wacc_add8(WAcc &a, const double (&l)[kItems],
                                          const bool (&in)[kItems])
{
    double x[kItems];
    bool up[kItems];
    double m = a.m;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        up[j] = in[j] && l[j] > m; // (false for NaN)
        x[j] = in[j] ? (up[j] ? m - l[j] : l[j] - m) : 0.0;
        m = up[j] ? l[j] : m;
    }
    // (-inf log-weights add nothing; x is -inf - -inf there and unused)
#pragma unroll
    for (int j = 0; j < kItems; ++j)
        x[j] = exp(x[j]);
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if (!in[j])
            continue;
        if (l[j] != l[j]) {
            a.s1 = l[j]; // NaN propagates to the degenerate check
        } else if (up[j]) {
            const double e = WAcc::one(l[j]);
            a.s1 = __dadd_rn(__dmul_rn(a.s1, x[j]), e);
            a.s2 = __fma_rn(e, e, __dmul_rn(a.s2, __dmul_rn(x[j], x[j])));
            a.m = l[j];
        } else if (l[j] > -INFINITY) {
            a.s1 = __dadd_rn(a.s1, x[j]);
            a.s2 = __fma_rn(x[j], x[j], a.s2);
        }
    }
}

__device__ __forceinline__ WAcc wacc_shfl_xor(const WAcc &a, int o)
{
    WAcc b;
    b.m = __shfl_xor_sync(0xffffffffu, a.m, o);
    b.s1 = __shfl_xor_sync(0xffffffffu, a.s1, o);
    b.s2 = __shfl_xor_sync(0xffffffffu, a.s2, o);
    return b;
}

// Shuffle tree per warp, then the warps in order; valid in thread 0.
__device__ __forceinline__ WAcc wacc_block(WAcc a, WAcc *sh)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        a.merge(wacc_shfl_xor(a, o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0)
        sh[wid] = a;
    __syncthreads();
    WAcc r = a;
    if (threadIdx.x == 0) {
        r = sh[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            r.merge(sh[w]);
    }
    return r;
}

// What a call sums (see k_weight_tiles).
enum {
    kWAdd = 0,       // lw (+ inc, stored): set_log_weight / add_log_weight
    kWEssLog = 1,    // ESS of w exp(inc): l = lw + inc
    kWEssLinear = 2, // b = w inc: sum |b|, sum b^2
    kWCessLog = 3,   // sum w e, sum w e e with e = exp(inc)
    kWCessLinear = 4 // ... with e = inc
};

// One tile's accumulator, before the block join; l: the log-weights.
template <int Kind>
__device__ __forceinline__ WAcc
weight_tile(long long N, long long base, double *lw, const double *w,
            const double *inc, double (&l)[kItems])
{
    constexpr bool Log = Kind == kWAdd || Kind == kWEssLog;
    double a[kItems], b[kItems];
    bool in[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const long long i = base + (long long)j * kThreads + threadIdx.x;
        in[j] = i < N;
        a[j] = in[j] ? (Log ? lw[i] : w[i]) : 0.0;
        b[j] = in[j] && inc != nullptr ? inc[i] : 0.0;
    }
    WAcc acc;
    if (Log) {
        acc.init(-INFINITY);
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            l[j] = inc != nullptr ? __dadd_rn(a[j], b[j]) : a[j];
        wacc_add8(acc, l, in);
    } else {
        acc.init(0.0); // plain sums: every partial has the same reference
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            if (Kind == kWEssLinear) {
                // the reference normalises by asum, a sum of |b|
                const double q = __dmul_rn(a[j], b[j]);
                if (in[j]) {
                    acc.s1 = __dadd_rn(acc.s1, fabs(q));
                    acc.s2 = __dadd_rn(acc.s2, __dmul_rn(q, q));
                }
            } else {
                const double e = Kind == kWCessLog ? exp(b[j]) : b[j];
                const double q = __dmul_rn(a[j], e);
                if (in[j]) {
                    acc.s1 = __dadd_rn(acc.s1, q);
                    acc.s2 = __dadd_rn(acc.s2, __dmul_rn(q, e));
                }
            }
        }
    }
    return acc;
}

__device__ __forceinline__ WeightCtl weight_result(const WAcc &r)
{
    WeightCtl c;
    c.M = r.m;
    c.S1 = r.s1;
    c.S2 = r.s2;
    c.error = (r.m > -INFINITY && r.m < INFINITY && r.s1 > 0.0 &&
               r.s1 < INFINITY)
                  ? 0
                  : (int)VSMC_CUDA_EDEGENERATE;
    return c;
}

template <int Kind>
__global__ void __launch_bounds__(kThreads)
k_weight_tiles(long long N, double *lw, const double *w, const double *inc,
               WAcc *tiles)
{
    __shared__ WAcc sh[kThreads / 32];
    const long long base = (long long)blockIdx.x * kTile;
    double l[kItems];
    const WAcc acc = weight_tile<Kind>(N, base, lw, w, inc, l);
    if (Kind == kWAdd && inc != nullptr) {
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const long long i = base + (long long)j * kThreads + threadIdx.x;
            if (i < N)
                lw[i] = l[j];
        }
    }
    const WAcc r = wacc_block(acc, sh);
    if (threadIdx.x == 0)
        tiles[blockIdx.x] = r;
}

// A thread's contiguous run of tiles.
__device__ __forceinline__ WAcc wacc_run(const WAcc *tiles, int b, int e)
{
    WAcc acc;
    acc.init(-INFINITY);
    for (int t = b; t < e; ++t) {
        const WAcc o = tiles[t];
        if (o.s1 != o.s1)
            acc.s1 = o.s1;
        else
            acc.merge(o);
    }
    return acc;
}

static __global__ void __launch_bounds__(kSpineThreads)
k_weight_join(const WAcc *tiles, int ntiles, WeightCtl *ctl, WeightCtl *out)
{
    __shared__ WAcc sh[kSpineThreads / 32];
    pdl_wait();
    const int per = (ntiles + blockDim.x - 1) / blockDim.x;
    const int b = threadIdx.x * per, e = min(b + per, ntiles);
    const WAcc r = wacc_block(wacc_run(tiles, b, e), sh);
    if (threadIdx.x == 0) {
        WeightCtl c = weight_result(r);
        *out = c;
        c.S2 = __ddiv_rn(1.0, c.S1); // the weights' coefficient
        *ctl = c;
    }
}

// lw += -max (normalize_log_weight); w = exp(lw) * (1 / sum).
static __global__ void __launch_bounds__(kThreads)
k_weight_apply(long long N, double *lw, double *w, const WeightCtl *ctl)
{
    pdl_wait();
    const double M = ctl->M, c = ctl->S2;
    const long long i0 =
        (long long)blockIdx.x * (4 * kThreads) + threadIdx.x;
    double l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (i0 + j * kThreads < N)
            l[j] = __dadd_rn(lw[i0 + j * kThreads], -M);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (i0 + j * kThreads < N) {
            lw[i0 + j * kThreads] = l[j];
            if (w != nullptr)
                w[i0 + j * kThreads] = __dmul_rn(exp(l[j]), c);
        }
}

// ---- up to 32 tiles: one cluster ------------------------------------------
constexpr int kWcCtas = 16;
constexpr int kWcTiles = 2 * kWcCtas;

struct WcShared {
    WAcc tile[2]; // this CTA's tiles (read by the other CTAs)
    WAcc sh[kThreads / 32];
    WeightCtl c;
};

// CTA c of the cluster holds tiles c and c + CTAs.
template <int Kind>
__global__ void __launch_bounds__(kThreads)
k_weight_cluster(long long N, double *lw, double *w, const double *inc,
                 WeightCtl *out)
{
    namespace cg = cooperative_groups;
    __shared__ WcShared sm;
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int nt = (int)((N + kTile - 1) / kTile);
    double l[2][kItems];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int t = rank + q * C;
        if (t < nt) {
            const WAcc r = wacc_block(
                weight_tile<Kind>(N, (long long)t * kTile, lw, w, inc, l[q]),
                sm.sh);
            if (threadIdx.x == 0)
                sm.tile[q] = r;
            __syncthreads();
        }
    }
    cl.sync();
    if (threadIdx.x < 32) {
        // the join's first warp (tile t in thread t; its other warps hold
        // none)
        const int t = threadIdx.x;
        WAcc a;
        a.init(-INFINITY);
        if (t < nt) {
            const WAcc o = cl.map_shared_rank(&sm, t % C)->tile[t / C];
            if (o.s1 != o.s1)
                a.s1 = o.s1;
            else
                a.merge(o);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            a.merge(wacc_shfl_xor(a, o));
        if (t == 0) {
            const WeightCtl c = weight_result(a);
            sm.c = c;
            if (rank == 0)
                *out = c;
        }
    }
    cl.sync(); // (also: no CTA leaves while another reads its tiles)
    if (Kind != kWAdd)
        return;
    const double M = sm.c.M, coeff = __ddiv_rn(1.0, sm.c.S1);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int t = rank + q * C;
        if (t >= nt)
            continue;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const long long i = (long long)t * kTile +
                                (long long)j * kThreads + threadIdx.x;
            if (i < N) {
                const double v = __dadd_rn(l[q][j], -M);
                lw[i] = v;
                if (w != nullptr)
                    w[i] = __dmul_rn(exp(v), coeff);
            }
        }
    }
}

} // namespace vsmc_b200
