// resample_cluster.cuh -- one resampling of a small filter in one launch.
//
// The pipeline of resample.cuh takes 5 to 14 launches.  For a filter of a
// few tiles each of them holds one or a few CTAs' work and costs 4 to 15 us
// of latency: kernel boundary, control block, global-memory round trips
// between producer and consumer.  Here one thread-block cluster runs the
// whole resampling: each group of kThreads threads owns one tile and keeps
// its weights, records and counts in registers; what tiles exchange (tile
// sums, exact-scan records and specials, zero counts, surplus prefixes)
// goes through distributed shared memory between cluster barriers; every
// CTA walks the exact scan redundantly (32 tiles, a few dozen specials), so
// no result has to be sent back.  Only a drawn U01 sequence goes through
// global memory (L2).  A cluster of up to 16 CTAs with two groups each
// covers kRcMaxTiles tiles (65536 particles).
//
// The results are those of the launch sequence: the exact scans reproduce
// the reference's sequential sums bit for bit whatever the split, and the
// mixed form's plain scan and residual sums keep the same association
// (the same block scans over the same 256 threads).
//
// Bound: latency (barriers, dependent shared-memory and L2 reads).
// Measured on one B200, us a step of a filter, launch sequence -> cluster:
// see launch_resample below.
#pragma once

#include <cooperative_groups.h>
#include <type_traits>

#include "resample.cuh"

namespace vsmc_b200 {

namespace cg = cooperative_groups;

constexpr int kRcMaxCtas = 16;  // CTAs of a cluster (above 8: non-portable)
constexpr int kRcGroups = 2;    // groups (tiles) of a CTA, at most
constexpr int kRcMaxTiles = kRcMaxCtas * kRcGroups;
constexpr int kRcStage = 256;   // specials of a scan staged per CTA

// How a resampling draws its U01 sequence.
enum { kRcSorted = 0, kRcStrat = 1, kRcSys = 2 };

// Barrier of one group (named barriers 1, 2; 0 is __syncthreads).
__device__ __forceinline__ void rc_gsync(int grp)
{
    asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(kThreads) : "memory");
}

struct RcScan {
    ExactTile tile;
    ExactSpecial spec[kExactCap];
};

// One group's shared memory; the first part is read by other CTAs.  The
// tile's scans: kRcU the sequence's terms, kRcA and kRcB the weights'
// scans in turn (normalisation, residuals' sum, weights), so that a CTA
// still reading one scan's records never meets the next one's.
enum { kRcA = 0, kRcB = 1, kRcU = 2 };

struct alignas(16) RcGroup {
    RcScan scan[3];
    double sum_w, sum_u;     // tile sums
    long long ksum;          // floor(N w) of the tile (residual)
    unsigned long long fixed; // the plain scan's tile total
    int zeros, sinc_last;
    alignas(16) int32_t sinc[kTile]; // surplus counts (sinc_local)
    // the group's own
    double sv_w[kExactCap], sv_u[kExactCap]; // exact S at the specials
    double red_d[kThreads / 32];
    unsigned long long red_k[kThreads / 32], red_s[kThreads / 32];
    int red_n[kThreads / 32], red_e[kThreads / 32];
    long long bound[2];
    alignas(16) double buf[kUStage]; // uniforms; overflow tiles' S; ranks
};

// The gathered records of one exact scan and its walk.
struct RcWalk {
    ExactTile t[kRcMaxTiles];
    int off[kRcMaxTiles + 1];
    double start[kRcMaxTiles + 1];
    ExactSpecial st[kRcStage];
    int overflow;
};

struct RcShared {
    RcWalk w, u;
    double sums[kRcMaxTiles], usums[kRcMaxTiles];
    double sh[kThreads / 32];
    double total; // the residuals' approximate sum
    long long NN;
    long long kexcl[kRcMaxTiles + 1];
    int zexcl[kRcMaxTiles + 1], E[kRcMaxTiles];
    double u0, delta;
    int kbits;
    unsigned long long offset;
    RcGroup g[1]; // as many as the CTA has groups
};

inline size_t rc_smem_bytes(int groups)
{
    return sizeof(RcShared) + (size_t)(groups - 1) * sizeof(RcGroup);
}

struct RcArgs {
    long long N;      // weights
    int nt;           // their tiles
    int cfrp;         // copy_from too (0: the counts only)
    int spine_done;   // tile_excl, NN, delta, kbits and u0 are set (filters)
    ResampleCtl *ctl;
    EngineRef eng;
    const double *tile_excl;
    double *u;        // the U01 sequence and its bins
    int32_t *bins;
    double *rec;      // an overflow tile's weights
    int32_t *rep_out;
    int32_t *copy_from;
};

// Exclusive scan over a group: block_excl_scan's association.
__device__ __forceinline__ double rc_excl_scan(double v, double *sh, int gtid,
                                               int grp, double &total)
{
    constexpr int NW = kThreads / 32;
    const int lane = gtid & 31, wid = gtid >> 5;
    const double inc = warp_incl_scan(v);
    if (lane == 31)
        sh[wid] = inc;
    rc_gsync(grp);
    if (wid == 0) {
        double s = lane < NW ? sh[lane] : 0.0;
        s = warp_incl_scan(s);
        if (lane < NW)
            sh[lane] = s;
    }
    rc_gsync(grp);
    const double wexcl = wid > 0 ? sh[wid - 1] : 0.0;
    total = sh[NW - 1];
    rc_gsync(grp);
    return wexcl + inc - v;
}

// ... of integers (any association).
template <typename T>
__device__ __forceinline__ T rc_excl_scan_int(T v, T *sh, int gtid, int grp,
                                              T &total)
{
    constexpr int NW = kThreads / 32;
    const int lane = gtid & 31, wid = gtid >> 5;
    const T inc = warp_incl_scan(v);
    if (lane == 31)
        sh[wid] = inc;
    rc_gsync(grp);
    T before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const T x = sh[w];
        before += w < wid ? x : T(0);
        all += x;
    }
    total = all;
    rc_gsync(grp);
    return before + inc - v;
}

// A thread's share of an exact scan: its element records (exact_scan.cuh)
// and the specials of the tile before them.
struct RcRec {
    double rec[kItems];
    int rank0;
};

// Classification of the group's tile (weights w, approximate start a and
// exclusive prefix pre): the tile's record and specials into `out`, the
// thread's records into r.  One segmented scan gives the clean k, the
// number of specials and the clean k since the last special before the
// thread's elements.
__device__ __forceinline__ void
rc_classify(long long base, long long N, const double (&w)[kItems], double a,
            double pre, double rel, int gtid, int grp, RcGroup &g,
            RcScan &out, double *dump, RcRec &r)
{
    constexpr int NW = kThreads / 32;
    const int lane = gtid & 31, wid = gtid >> 5;
    const long long i0 = base + (long long)gtid * kItems;
    ExactLocal x;
    exact_classify(i0, N, w, a, pre, rel, x);
    const unsigned long long kr = x.kloc[kItems - 1];
    unsigned long long kat = 0; // kloc at the thread's last special
#pragma unroll
    for (int j = 0; j < kItems; ++j)
        if ((x.special >> j) & 1u)
            kat = x.kloc[j];
    unsigned long long k = kr, s = x.nsp ? kr - kat : kr;
    int n = x.nsp;
    const int elast =
        (x.special >> (kItems - 1)) & 1u ? kNoBinade : x.e[kItems - 1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long pk = __shfl_up_sync(0xffffffffu, k, o);
        const unsigned long long ps = __shfl_up_sync(0xffffffffu, s, o);
        const int pn = __shfl_up_sync(0xffffffffu, n, o);
        if (lane >= o) {
            k += pk;
            s = n ? s : ps + s;
            n += pn;
        }
    }
    if (lane == 31) {
        g.red_k[wid] = k;
        g.red_s[wid] = s;
        g.red_n[wid] = n;
        g.red_e[wid] = elast;
    }
    // exclusive within the warp
    unsigned long long ke = __shfl_up_sync(0xffffffffu, k, 1);
    unsigned long long se = __shfl_up_sync(0xffffffffu, s, 1);
    int ne = __shfl_up_sync(0xffffffffu, n, 1);
    int e_before = __shfl_up_sync(0xffffffffu, elast, 1);
    if (lane == 0) {
        ke = se = 0;
        ne = 0;
    }
    rc_gsync(grp);
    unsigned long long kp = 0, sp = 0, ktile = 0;
    int np = 0, nspec = 0;
#pragma unroll
    for (int q = 0; q < NW; ++q) {
        const unsigned long long qk = g.red_k[q];
        const int qn = g.red_n[q];
        if (q < wid) {
            kp += qk;
            sp = qn ? g.red_s[q] : sp + g.red_s[q];
            np += qn;
        }
        ktile += qk;
        nspec += qn;
    }
    if (lane == 0)
        e_before = wid > 0 ? g.red_e[wid - 1] : kNoBinade;
    ke += kp;
    se = ne ? se : sp + se;
    r.rank0 = np + ne;
    const long long last = min(base + (long long)kTile, N) - 1;
    int rank = r.rank0;
    unsigned long long kb = 0; // kloc at the last special, se before it
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if ((x.special >> j) & 1u) {
            if (rank < kExactCap) {
                ExactSpecial q;
                q.w = w[j];
                q.k_before = ke + x.kloc[j];
                q.idx = (int)(i0 + j - base);
                q.e_seg = j == 0 ? e_before
                                 : ((x.special >> (j - 1)) & 1u
                                        ? kNoBinade
                                        : x.e[j - 1]);
                out.spec[rank] = q;
            }
            ++rank;
            se = 0;
            kb = x.kloc[j];
            r.rec[j] = -1.0;
        } else {
            const unsigned long long K = se + (x.kloc[j] - kb);
            r.rec[j] = K == 0 ? 0.0
                              : __dmul_rn((double)K, exact_pow2(x.e[j] - 52));
        }
        if (i0 + j == last)
            out.tile.e_last = (x.special >> j) & 1u ? kNoBinade : x.e[j];
    }
    if (gtid == 0) {
        out.tile.k_total = ktile;
        out.tile.nspec = nspec;
    }
    // a tile with more specials than kept: its values for the walk
    if (nspec > kExactCap) {
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            if (i0 + j < N)
                dump[i0 + j] = w[j];
    }
    rc_gsync(grp); // the red_* arrays are free again
}

// The records of every tile's scan into the CTA's shared memory (after the
// cluster barrier): warp `wq` reads the tile records, then all threads the
// specials (a CTA barrier between them).
template <int B>
__device__ __forceinline__ void rc_gather_tiles(cg::cluster_group &cl,
                                                RcShared &sm, RcWalk &k,
                                                int nt, int G, int wq)
{
    const int lane = threadIdx.x & 31;
    if ((int)(threadIdx.x >> 5) == wq) {
        ExactTile et;
        et.k_total = 0;
        et.nspec = 0;
        et.e_last = kNoBinade;
        if (lane < nt) {
            const RcGroup *rg = cl.map_shared_rank(&sm.g[lane % G], lane / G);
            et = rg->scan[B].tile;
        }
        k.t[lane] = et;
        const int ns = et.nspec <= kExactCap ? et.nspec : 0;
        const int in = warp_incl_scan(ns);
        k.off[lane] = in - ns;
        if (lane == 31)
            k.off[32] = in;
        const unsigned ov = __ballot_sync(0xffffffffu, et.nspec > kExactCap);
        if (lane == 0)
            k.overflow = ov != 0;
    }
}

template <int B>
__device__ __forceinline__ void rc_gather_specials(cg::cluster_group &cl,
                                                   RcShared &sm, RcWalk &k,
                                                   int nt, int G)
{
    if (k.off[32] > kRcStage)
        return;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int t = threadIdx.x >> 5; t < nt; t += nw) {
        const int b = k.off[t], n = k.off[t + 1] - b;
        if (n == 0)
            continue;
        const RcGroup *rg = cl.map_shared_rank(&sm.g[t % G], t / G);
        const ExactSpecial *sp = rg->scan[B].spec;
        for (int r = lane; r < n; r += 32)
            k.st[b + r] = sp[r];
    }
}

// Phase B of the exact scan (one thread): the exact S before every tile
// and, for the CTA's own tiles [own, own + G), at their specials.
// Overflow tiles are summed element by element from `vals`; their S goes
// into the group's buffer.
template <int B>
__device__ __forceinline__ void rc_walk(cg::cluster_group &cl, RcShared &sm,
                                        RcWalk &k, int nt, int G, int own,
                                        const double *vals, long long N)
{
    constexpr bool U = B == kRcU;
    const bool fits = k.off[32] <= kRcStage;
    double S = 0.0;
    for (int t = 0; t < nt; ++t) {
        k.start[t] = S;
        const ExactTile et = k.t[t];
        const int mine = t - own;
        const bool keep = mine >= 0 && mine < G;
        if (et.nspec <= kExactCap) {
            unsigned long long kb = 0;
            for (int r = 0; r < et.nspec; ++r) {
                ExactSpecial sp;
                if (fits) {
                    sp = k.st[k.off[t] + r];
                } else {
                    const RcGroup *rg =
                        cl.map_shared_rank(&sm.g[t % G], t / G);
                    sp = rg->scan[B].spec[r];
                }
                const unsigned long long seg = sp.k_before - kb;
                if (seg != 0)
                    S = __dadd_rn(S, __dmul_rn((double)seg,
                                               exact_pow2(sp.e_seg - 52)));
                S = __dadd_rn(S, sp.w);
                if (keep) {
                    if (U)
                        sm.g[mine].sv_u[r] = S;
                    else
                        sm.g[mine].sv_w[r] = S;
                }
                kb = sp.k_before;
            }
            const unsigned long long tail = et.k_total - kb;
            if (tail != 0)
                S = __dadd_rn(S, __dmul_rn((double)tail,
                                           exact_pow2(et.e_last - 52)));
        } else {
            const long long b0 = (long long)t * kTile;
            const int n = (int)(min(b0 + (long long)kTile, N) - b0);
            double *out = keep ? sm.g[mine].buf + (U ? kTile : 0) : nullptr;
            for (int i = 0; i < n; ++i) {
                S = __dadd_rn(S, vals[b0 + i]);
                if (keep)
                    out[i] = S;
            }
        }
    }
    k.start[nt] = S;
}

// The exact S of a thread's elements after the walk.
template <bool U>
__device__ __forceinline__ void rc_values(const RcShared &sm, const RcWalk &k,
                                          const RcGroup &g, int tile,
                                          int gtid, const RcRec &r,
                                          double (&S)[kItems])
{
    if (k.t[tile].nspec > kExactCap) {
        const double *o = g.buf + (U ? kTile : 0) + gtid * kItems;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            S[j] = o[j];
        return;
    }
    exact_values(r.rec, r.rank0, k.start[tile], U ? g.sv_u : g.sv_w, false,
                 S);
}

// Sum of the tile sums before tile t (for the classification).
__device__ __forceinline__ double rc_before(const double *sums, int t)
{
    double a = 0.0;
    for (int q = 0; q < t; ++q)
        a += sums[q];
    return a;
}

// Eight consecutive values of a thread (zero past N).
template <typename T>
__device__ __forceinline__ void rc_load8(const T *src, long long i0,
                                         long long N, T (&v)[kItems])
{
    if (i0 + kItems <= N &&
        (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        constexpr int P = 16 / sizeof(T);
#pragma unroll
        for (int j = 0; j < kItems / P; ++j) {
            const int4 q =
                *reinterpret_cast<const int4 *>(src + i0 + j * P);
            const T *t = reinterpret_cast<const T *>(&q);
#pragma unroll
            for (int m = 0; m < P; ++m)
                v[j * P + m] = t[m];
        }
    } else {
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            v[j] = i0 + j < N ? src[i0 + j] : T(0);
    }
}

// Eight consecutive ints to a caller's array of any alignment.
__device__ __forceinline__ void rc_store8(int32_t *dst, long long i0,
                                          long long N,
                                          const int (&v)[kItems])
{
    if (i0 + kItems <= N && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        int4 *d = reinterpret_cast<int4 *>(dst + i0);
        d[0] = make_int4(v[0], v[1], v[2], v[3]);
        d[1] = make_int4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            if (i0 + j < N)
                dst[i0 + j] = v[j];
    }
}

// One resampling; every thread of the cluster calls it.
template <typename W, bool Residual, int U>
__device__ __forceinline__ void rc_resample(W wsrc, const RcArgs &a,
                                            RcShared &sm)
{
    constexpr bool Sys = U == kRcSys;
    constexpr int NW = kThreads / 32;
    if (!a.ctl->active)
        return; // (the whole cluster)
    cg::cluster_group cl = cg::this_cluster();
    const int G = (int)blockDim.x / kThreads;
    const int rank = (int)cl.block_rank();
    const int grp = (int)threadIdx.x / kThreads;
    const int gtid = (int)threadIdx.x % kThreads;
    const int lane = gtid & 31, wid = gtid >> 5;
    const int own = rank * G;
    const int tile = own + grp;
    const int nt = a.nt;
    const long long N = a.N;
    RcGroup &g = sm.g[grp];
    const bool act = tile < nt;
    const long long base = (long long)tile * kTile;
    const long long i0 = base + (long long)gtid * kItems;
    const long long Nout = resample_children(a.ctl, N);
    const double Nd = (double)Nout;
    wsrc.prepare();
    if (threadIdx.x == 0) {
        const ResampleCtl *c = a.ctl;
        sm.offset = c->offset;
        if (a.spine_done && !Residual) {
            sm.NN = c->NN;
            sm.delta = c->delta;
            sm.kbits = c->kbits;
            sm.u0 = Sys ? c->u0 : 0.0;
        } else if (!Residual) {
            sm.NN = Nout;
            sm.delta = __ddiv_rn(1.0, Nd);
            sm.kbits = bin_kbits(Nout);
            sm.u0 = Sys ? __dmul_rn(canonical_u64(threefry_word(
                                        a.eng.key, a.eng.ctr, c->offset)),
                                    sm.delta)
                        : 0.0;
        }
        if (rank == 0)
            a.ctl->words = Sys ? 1 : 0;
    }
    __syncthreads();

    // ---- the weights --------------------------------------------------
    double w[kItems]; // as scanned
    int kk[kItems];   // floor(N w) (residual)
    RcRec rw;
    double pre = 0.0, coeff_r = 1.0;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        w[j] = 0.0;
        kk[j] = 0;
    }
    if (act) {
        typename W::stage_t x[kItems];
        rc_load8(wsrc.stage_src(), i0, N, x);
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            if (i0 + j < N)
                w[j] = W::kExactNorm ? wsrc.unnorm_stage(x[j])
                                     : wsrc.from_stage(x[j]);
    }
    if (W::kExactNorm) {
        // the sequential sum of exp(lw - M); its reciprocal normalises
        if (act) {
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < kItems; ++j)
                run += w[j];
            pre = rc_excl_scan(run, g.red_d, gtid, grp, total);
            rc_classify(base, N, w,
                        __dmul_rn(a.tile_excl[tile], wsrc.spine_unnorm()),
                        pre, ExactMargin<W>::rel, gtid, grp, g, g.scan[kRcA], a.rec,
                        rw);
        }
    }
    // the drawn sequence's first stage, beside the weights' (its length is
    // known unless the scheme is residual)
    double tv[kItems]; // negated terms
    RcRec ru;
    double pre_u = 0.0;
    const auto terms = [&]() {
        // log(1 - U_n) / (NN - n), negated, and the tile's sum
        const long long NN = sm.NN;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            tv[j] = 0.0;
        if (base < NN) {
            if (i0 < NN) {
                sorted_terms8(a.eng, sm.offset, i0, NN, tv);
#pragma unroll
                for (int j = 0; j < kItems; ++j)
                    tv[j] = -tv[j];
            }
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < kItems; ++j)
                run += tv[j];
            pre_u = rc_excl_scan(run, g.red_d, gtid, grp, total);
            if (gtid == 0)
                g.sum_u = total;
        }
    };
    const auto utiles = [&]() {
        return (int)min((sm.NN + kTile - 1) / kTile, (long long)kRcMaxTiles);
    };
    const auto terms_classify = [&]() {
        // (the terms' tile sums are in sm.usums)
        if (base < sm.NN)
            rc_classify(base, sm.NN, tv, rc_before(sm.usums, tile), pre_u,
                        ExactMargin<TermsNeg>::rel, gtid, grp, g,
                        g.scan[kRcU], a.u,
                        ru);
    };
    const auto gather_usums = [&](int nu) {
        if ((int)(threadIdx.x >> 5) == NW - 1 && lane < nu)
            sm.usums[lane] =
                cl.map_shared_rank(&sm.g[lane % G], lane / G)->sum_u;
    };
    // u_n = 1 - exp(lmax_n), its running maximum and the bin index
    const auto sorted_values = [&]() {
        const long long NN = sm.NN;
        if (base >= NN)
            return;
        double S[kItems];
        rc_values<true>(sm, sm.u, g, tile, gtid, ru, S);
        const double s0 = sm.u.start[tile];
        const double umax =
            tile > 0 ? __dadd_rn(1.0, -fm::fm_exp(-s0)) : -INFINITY;
        double uv[kItems];
        double tmax = -INFINITY;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            uv[j] = __dadd_rn(1.0, -fm::fm_exp(-S[j]));
            tmax = fmax(tmax, uv[j]);
        }
        double inc = tmax;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o)
                inc = fmax(inc, v);
        }
        if (lane == 31)
            g.red_d[wid] = inc;
        double exc = __shfl_up_sync(0xffffffffu, inc, 1);
        if (lane == 0)
            exc = -INFINITY;
        rc_gsync(grp);
        for (int q = 0; q < wid; ++q)
            exc = fmax(exc, g.red_d[q]);
        rc_gsync(grp);
        double m = fmax(umax, exc);
        const int kb = sm.kbits;
        long long kprev = bin_floor(m, kb);
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            m = fmax(m, uv[j]);
            const long long n = i0 + j;
            if (n < NN) {
                a.u[n] = m;
                const long long khi = bin_floor(m, kb);
                bin_fill(a.bins, kb, n == 0 ? 0 : kprev + 1, khi, n, NN);
                kprev = khi;
            }
        }
    };
    // the stratified sequence (k_uniforms_stratified_body's values)
    const auto strat_values = [&]() {
        const long long NN = sm.NN;
        if (base >= NN)
            return;
        const double delta = sm.delta;
        const int kb = sm.kbits;
        const unsigned long long off = sm.offset;
        double raw[kItems];
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            raw[j] = -INFINITY;
        if (i0 < NN) {
            uint64_t q[8];
            threefry_words8(a.eng, off + (unsigned long long)i0, q);
#pragma unroll
            for (int j = 0; j < kItems; ++j)
                if (i0 + j < NN)
                    raw[j] = strat_u(q[j], i0 + j, delta);
        }
        double p1 = __shfl_up_sync(0xffffffffu, raw[7], 1);
        double p2 = __shfl_up_sync(0xffffffffu, raw[6], 1);
        if (lane == 31) {
            g.red_d[wid] = raw[7];
            g.sv_u[wid] = raw[6];
        }
        rc_gsync(grp);
        if (lane == 0) {
            p1 = p2 = -INFINITY;
            if (wid > 0) {
                p1 = g.red_d[wid - 1];
                p2 = g.sv_u[wid - 1];
            } else if (base > 0) {
                p1 = strat_u(threefry_word(a.eng.key, a.eng.ctr,
                                           off + i0 - 1),
                             i0 - 1, delta);
                p2 = strat_u(threefry_word(a.eng.key, a.eng.ctr,
                                           off + i0 - 2),
                             i0 - 2, delta);
            }
        }
        rc_gsync(grp);
        long long kprev = bin_floor(fmax(p1, p2), kb);
        double rprev = p1;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const long long n = i0 + j;
            if (n < NN) {
                const double v = fmax(raw[j], rprev);
                a.u[n] = v;
                const long long khi = bin_floor(v, kb);
                bin_fill(a.bins, kb, n == 0 ? 0 : kprev + 1, khi, n, NN);
                kprev = khi;
            }
            rprev = raw[j];
        }
    };
    // the walks of the weights' and / or the terms' scans (after a cluster
    // barrier); a walk over an overflow tile reads its values in global
    // memory, and one over more specials than staged reads the other CTAs',
    // which their owners reuse afterwards
    const auto walks = [&](auto buf, bool ww, bool wu) {
        constexpr int B = decltype(buf)::value;
        const int nu = wu ? utiles() : 0;
        if (ww)
            rc_gather_tiles<B>(cl, sm, sm.w, nt, G, 0);
        if (wu)
            rc_gather_tiles<kRcU>(cl, sm, sm.u, nu, G, 1);
        __syncthreads();
        if (ww)
            rc_gather_specials<B>(cl, sm, sm.w, nt, G);
        if (wu)
            rc_gather_specials<kRcU>(cl, sm, sm.u, nu, G);
        __syncthreads();
        if (ww && threadIdx.x == 0)
            rc_walk<B>(cl, sm, sm.w, nt, G, own, a.rec, N);
        if (wu && threadIdx.x == 32)
            rc_walk<kRcU>(cl, sm, sm.u, nu, G, own, a.u, sm.NN);
        __syncthreads();
        if ((ww && (sm.w.overflow || sm.w.off[32] > kRcStage)) ||
            (wu && (sm.u.overflow || sm.u.off[32] > kRcStage)))
            cl.sync();
    };

    if (!Residual) {
        if (U == kRcStrat)
            strat_values();
        if (U == kRcSorted)
            terms();
    }
    if (W::kExactNorm) {
        cl.sync();
        if (!Residual && U == kRcSorted)
            gather_usums(utiles());
        walks(std::integral_constant<int, kRcA>(), true, false);
        // w = exp(lw - M) * (1 / sum)
        const double coeff = __ddiv_rn(1.0, sm.w.start[nt]);
        pre *= coeff;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            w[j] = __dmul_rn(w[j], coeff);
    }
    bool exact = true;
    if (Residual) {
        // r = modf(N w, &k); the tile's sums
        double r[kItems];
        long long ks = 0;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            double k = 0.0;
            r[j] = i0 + j < N ? residual_split(w[j], Nd, k) : 0.0;
            kk[j] = (int32_t)k;
            ks += (long long)k;
        }
        if (act) {
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < kItems; ++j)
                run += fabs(r[j]);
            if (W::kApprox) {
                // the launch sequence's sum: strided elements per thread,
                // warp trees, the warps in order
                double s = 0.0;
#pragma unroll
                for (int j = 0; j < kItems; ++j)
                    g.buf[pad8(gtid * kItems + j)] = fabs(r[j]);
                rc_gsync(grp);
#pragma unroll
                for (int j = 0; j < kItems; ++j) {
                    const int l = j * kThreads + gtid;
                    if (base + l < N)
                        s += g.buf[pad8(l)];
                }
                s = warp_sum(s);
                if (lane == 0)
                    g.red_d[wid] = s;
                rc_gsync(grp);
                if (gtid == 0) {
                    double t = 0.0;
                    for (int q = 0; q < NW; ++q)
                        t += g.red_d[q];
                    g.sum_w = t;
                }
                rc_gsync(grp);
            } else {
                pre = rc_excl_scan(run, g.red_d, gtid, grp, total);
                if (gtid == 0)
                    g.sum_w = total;
            }
            long long kt;
            rc_excl_scan_int(ks, reinterpret_cast<long long *>(g.red_k), gtid,
                             grp, kt);
            if (gtid == 0)
                g.ksum = kt;
        }
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            w[j] = r[j];
        cl.sync();
        // NN = children - sum floor(N w); the residuals' approximate sum
        if (threadIdx.x < 32) {
            long long k = 0;
            if (lane < nt) {
                const RcGroup *rg =
                    cl.map_shared_rank(&sm.g[lane % G], lane / G);
                k = rg->ksum;
                sm.sums[lane] = rg->sum_w;
            }
            const long long ki = warp_incl_scan(k);
            sm.kexcl[lane] = ki - k;
            if (lane == 31)
                sm.kexcl[32] = ki;
            __syncwarp();
            // (spine of at most 256 tiles on 256 threads: tile t in thread
            // t, so the total is the first warp's inclusive scan, then the
            // scan of the warps' totals, of which only the first is not 0)
            double x = lane < nt ? sm.sums[lane] : 0.0;
            x = warp_incl_scan(x);
            if (lane == 31) {
                sm.total = x;
                const long long NN = Nout - ki;
                sm.NN = NN;
                sm.delta = __ddiv_rn(1.0, (double)NN);
                sm.kbits = bin_kbits(NN);
                sm.u0 = 0.0;
                if (Sys)
                    sm.u0 = __dmul_rn(canonical_u64(threefry_word(
                                          a.eng.key, a.eng.ctr, sm.offset)),
                                      sm.delta);
            }
        }
        __syncthreads();
        exact = sm.NN > 0;
        if (exact) {
            if (U == kRcStrat)
                strat_values();
            if (U == kRcSorted)
                terms();
        }
        if (!W::kApprox && exact) {
            // the residuals' sequential sum
            const double a0 = act ? rc_before(sm.sums, tile) : 0.0;
            if (act)
                rc_classify(base, N, w, a0, pre, ExactMargin<W>::rel, gtid,
                            grp, g, g.scan[kRcB], a.rec, rw);
            cl.sync();
            if (U == kRcSorted) {
                gather_usums(utiles());
                __syncthreads();
            }
            walks(std::integral_constant<int, kRcB>(), true, false);
            coeff_r = __ddiv_rn(1.0, sm.w.start[nt]);
            if (act) {
                pre *= coeff_r;
#pragma unroll
                for (int j = 0; j < kItems; ++j)
                    w[j] = __dmul_rn(w[j], coeff_r);
                rc_classify(base, N, w, a0 * coeff_r, pre,
                            ExactMargin<W>::rel, gtid, grp, g, g.scan[kRcA], a.rec,
                            rw);
            }
        } else if (W::kApprox) {
            coeff_r = __ddiv_rn(1.0, sm.total);
#pragma unroll
            for (int j = 0; j < kItems; ++j)
                w[j] = __dmul_rn(w[j], coeff_r);
        }
    } else if (W::kExactNorm) {
        if (act)
            rc_classify(base, N, w,
                        __dmul_rn(a.tile_excl[tile],
                                  __ddiv_rn(wsrc.spine_unnorm(),
                                            sm.w.start[nt])),
                        pre, ExactMargin<W>::rel, gtid, grp, g, g.scan[kRcB], a.rec,
                        rw);
    } else if (!W::kApprox) {
        // given weights: tile sums first
        if (act) {
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < kItems; ++j)
                run += w[j];
            pre = rc_excl_scan(run, g.red_d, gtid, grp, total);
            if (gtid == 0)
                g.sum_w = total;
        }
        cl.sync();
        if (threadIdx.x < 32 && lane < nt)
            sm.sums[lane] =
                cl.map_shared_rank(&sm.g[lane % G], lane / G)->sum_w;
        if (U == kRcSorted)
            gather_usums(utiles());
        __syncthreads();
        if (act)
            rc_classify(base, N, w, rc_before(sm.sums, tile), pre,
                        ExactMargin<W>::rel, gtid, grp, g, g.scan[kRcA], a.rec, rw);
    }
    if (W::kApprox && exact && act) {
        // the plain scan: inclusive prefixes within the tile, the tile's
        // total in fixed point
        double run = 0.0, total;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            run += w[j];
        double s = rc_excl_scan(run, g.red_d, gtid, grp, total);
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            s += w[j];
            rw.rec[j] = s;
        }
        if (gtid == 0)
            g.fixed = approx_fixed(total);
    }
    if (W::kApprox && U == kRcSorted && exact) {
        cl.sync();
        gather_usums(utiles());
        __syncthreads();
    }
    if (U == kRcSorted && exact)
        terms_classify();
    cl.sync();

    // ---- the cumulative weights ------------------------------------------
    double Cx[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j)
        Cx[j] = 0.0;
    if (exact) {
        // the weights' scan: kRcB after the normalisation's, else kRcA
        constexpr int B = !Residual && W::kExactNorm ? kRcB : kRcA;
        walks(std::integral_constant<int, B>(), !W::kApprox,
              U == kRcSorted);
        if (W::kApprox) {
            if (threadIdx.x < 32) {
                unsigned long long f = 0;
                if (lane < nt)
                    f = cl.map_shared_rank(&sm.g[lane % G], lane / G)->fixed;
                const unsigned long long fi = warp_incl_scan(f);
                sm.w.start[lane] =
                    __dmul_rn(__ull2double_rn(fi - f), 1.0 / kApproxScale);
                if (lane == 31)
                    sm.w.start[32] =
                        __dmul_rn(__ull2double_rn(fi), 1.0 / kApproxScale);
            }
            __syncthreads();
            if (act) {
                const double s0 = sm.w.start[tile];
#pragma unroll
                for (int j = 0; j < kItems; ++j)
                    Cx[j] = __dadd_rn(s0, rw.rec[j]);
            }
        } else if (act) {
            rc_values<false>(sm, sm.w, g, tile, gtid, rw, Cx);
        }
        if (U == kRcSorted) {
            sorted_values();
            cl.sync();
        }
    }

    // ---- inversion ---------------------------------------------------
    const long long NN = sm.NN;
    const double u0 = sm.u0, delta = sm.delta;
    const long long nu = NN;
    const double *u = a.u;
    double *sw = g.buf;
    int rep[kItems];
    int zl[kItems]; // rank among the tile's slots without offspring, or -1
    if (act) {
        const double sa = exact ? sm.w.start[tile] : 0.0;
        const double sb = exact ? sm.w.start[tile + 1] : 0.0;
        if (wid < 2) {
            const double C = wid == 0 ? sa : sb;
            long long r;
            if ((wid == 0 && tile == 0) || nu <= 0) {
                r = 0;
            } else if (Sys) {
                r = sys_count(C, u0, delta, NN);
            } else {
                long long wl, wh;
                bin_window(a.bins, sm.kbits, nu, C, wl, wh);
                wl = max(min(wl, nu), 0ll);
                wh = min(max(wh, wl), nu);
                r = warp_upper_bound([u](long long i) { return u[i]; }, wl,
                                     wh, C);
            }
            if (lane == 0)
                g.bound[wid] = r;
        }
        rc_gsync(grp);
        const long long lo = g.bound[0];
        const long long hi = max(g.bound[1], lo);
        const bool staged = !Sys && (hi - lo) <= kUStage;
        if (staged) {
            for (int k = gtid; k < (int)(hi - lo); k += kThreads)
                cp_async8(&sw[k], &u[lo + k]);
            cp_async_commit();
            cp_async_wait_all();
        }
        rc_gsync(grp);
        const int ilo = (int)lo, ihi = (int)hi, iNN = (int)NN, iN = (int)N;
        const int p0 = (int)i0;
        const int tile_last = (int)min(base + (long long)kTile, N) - 1;
        int cnt[kItems];
        int pos = -1;
        long long gpos = -1;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const int i = p0 + j;
            const double C = Cx[j];
            int c;
            if (i >= iN - 1) {
                c = iNN; // the last particle takes every remaining uniform
            } else if (W::kApprox && i == tile_last) {
                c = ihi; // the plain scan: closes at the next tile's start
            } else if (Sys) {
                c = (int)sys_count(C, u0, delta, NN);
            } else if (staged) {
                pos = pos < 0 ? ub_shared(sw, 0, ihi - ilo, C)
                              : ub_gallop(sw, pos, ihi - ilo, C);
                c = ilo + pos;
            } else {
                gpos = gpos < 0 ? ub_global(u, lo, hi, C)
                                : ub_gallop_global(u, gpos, hi, C);
                c = (int)gpos;
            }
            cnt[j] = min(max(c, ilo), i >= iN - 1 ? iNN : ihi);
        }
#pragma unroll
        for (int j = 1; j < kItems; ++j)
            cnt[j] = max(cnt[j], cnt[j - 1]);
        int prev = __shfl_up_sync(0xffffffffu, cnt[kItems - 1], 1);
        if (lane == 31)
            g.red_e[wid] = cnt[kItems - 1];
        rc_gsync(grp);
        if (lane == 0)
            prev = wid == 0 ? (tile > 0 ? ilo : 0) : g.red_e[wid - 1];
        int zeros = 0, ksum = 0;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const int i = p0 + j;
            const int c = max(cnt[j], prev);
            rep[j] = (i < iN) ? (c - prev) + kk[j] : 0;
            prev = c;
            cnt[j] = c;
            zeros += (i < iN && rep[j] == 0) ? 1 : 0;
            ksum += kk[j];
            // the last queried uniform fixes the words drawn
            if (i == iN - 2 && !Sys)
                a.ctl->words =
                    NN > 0 ? (unsigned long long)min(iNN, c + 1) : 0ull;
            if (i == iN - 2)
                a.ctl->n_final = c;
        }
        int ztot, ktot;
        int zloc = rc_excl_scan_int(zeros, g.red_n, gtid, grp, ztot);
        int kprefix = 0;
        if (Residual)
            kprefix = (int)sm.kexcl[tile] +
                      rc_excl_scan_int(ksum, g.red_n, gtid, grp, ktot);
        if (gtid == 0)
            g.zeros = ztot;
        int sc[kItems];
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const int i = p0 + j;
            kprefix += kk[j];
            const int R = (i >= iN - 1) ? (int)Nout : cnt[j] + kprefix;
            zl[j] = -1;
            if (rep[j] == 0) {
                zl[j] = zloc;
                ++zloc;
            }
            sc[j] = R - (i + 1) + zloc;
            if (i == tile_last)
                g.sinc_last = sc[j];
        }
        int4 *sd = reinterpret_cast<int4 *>(g.sinc + gtid * kItems);
        sd[0] = make_int4(sc[0], sc[1], sc[2], sc[3]);
        sd[1] = make_int4(sc[4], sc[5], sc[6], sc[7]);
        if (a.rep_out != nullptr)
            rc_store8(a.rep_out, i0, N, rep);
    }
    cl.sync();
    if (rank == 0 && threadIdx.x == 0)
        a.ctl->offset += *(volatile unsigned long long *)&a.ctl->words;
    if (!a.cfrp)
        return;

    // ---- the slots without offspring (k_zero_spine, k_cfrp_fill) ---------
    if (threadIdx.x < 32) {
        int z = 0, sl = 0;
        if (lane < nt) {
            const RcGroup *rg = cl.map_shared_rank(&sm.g[lane % G], lane / G);
            z = rg->zeros;
            sl = rg->sinc_last;
        }
        const int zi = warp_incl_scan(z);
        sm.zexcl[lane] = zi - z;
        if (lane == 31)
            sm.zexcl[32] = zi;
        sm.E[lane] = sl + zi - z;
    }
    __syncthreads();
    if (act) {
        const int Z0 = sm.zexcl[tile];
        const int z = min(sm.zexcl[tile + 1] - Z0, kTile);
        int *tab = reinterpret_cast<int *>(g.buf); // z ranks (and kTile + 8)
        int top = 0; // ranks covered
        if (z > 0) {
            // the first tiles with E > Z0 and E > Z0 + z - 1
            const int e = lane < nt ? sm.E[lane] : INT_MAX;
            const unsigned above0 = __ballot_sync(0xffffffffu, e > Z0);
            const unsigned above1 =
                __ballot_sync(0xffffffffu, e > Z0 + z - 1);
            const int tf = min(__ffs(above0) - 1, nt - 1);
            const int tl = min(__ffs(above1) - 1, nt - 1);
            const int4 none = make_int4(-1, -1, -1, -1);
            int4 *t4 = reinterpret_cast<int4 *>(tab + gtid * kItems);
            t4[0] = none;
            t4[1] = none;
            rc_gsync(grp);
            // parent p owns the ranks [sinc(p - 1), sinc(p)): it marks the
            // first of them that falls in the window
            int prev_top = INT_MIN;
            for (int pt = tf; pt <= tl; ++pt) {
                const long long pb = (long long)pt * kTile;
                const int len = (int)min((long long)kTile, N - pb);
                const int zoff = sm.zexcl[pt];
                const RcGroup *rg = cl.map_shared_rank(&sm.g[pt % G], pt / G);
                const int4 *s4 =
                    reinterpret_cast<const int4 *>(rg->sinc + gtid * kItems);
                const int4 q0 = s4[0], q1 = s4[1];
                const int v[kItems] = {q0.x, q0.y, q0.z, q0.w,
                                       q1.x, q1.y, q1.z, q1.w};
                int before = gtid > 0 ? rg->sinc[gtid * kItems - 1] + zoff
                                      : prev_top;
#pragma unroll
                for (int j = 0; j < kItems; ++j) {
                    const int l = gtid * kItems + j;
                    if (l < len) {
                        const int cur = v[j] + zoff;
                        const int rl = max(before, Z0);
                        if (rl < min(cur, Z0 + z))
                            tab[rl - Z0] = (int)pb + l;
                        before = cur;
                    }
                }
                prev_top = max(prev_top, rg->sinc[len - 1] + zoff);
            }
            top = prev_top - Z0;
            rc_gsync(grp);
            // parents increase with the rank: the running maximum of the
            // marks is each rank's parent
            const int4 m0 = t4[0], m1 = t4[1];
            int m[kItems] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
            for (int j = 1; j < kItems; ++j)
                m[j] = max(m[j], m[j - 1]);
            int in = m[kItems - 1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int q = __shfl_up_sync(0xffffffffu, in, o);
                if (lane >= o)
                    in = max(in, q);
            }
            if (lane == 31)
                g.red_n[wid] = in;
            int ex = __shfl_up_sync(0xffffffffu, in, 1);
            if (lane == 0)
                ex = -1;
            rc_gsync(grp);
            for (int q = 0; q < wid; ++q)
                ex = max(ex, g.red_n[q]);
            t4[0] = make_int4(max(m[0], ex), max(m[1], ex), max(m[2], ex),
                              max(m[3], ex));
            t4[1] = make_int4(max(m[4], ex), max(m[5], ex), max(m[6], ex),
                              max(m[7], ex));
            rc_gsync(grp);
        }
        int cf[kItems];
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            cf[j] = (int)i0 + j;
            if (i0 + j < N && zl[j] >= 0) {
                const int p = zl[j] < min(z, top) ? tab[zl[j]] : -1;
                if (p >= 0)
                    cf[j] = p;
                else // no parent found: replication != N
                    atomicExch(&a.ctl->error, (int)VSMC_CUDA_EDEGENERATE);
            }
        }
        rc_store8(a.copy_from, i0, N, cf);
    }
    cl.sync(); // no CTA leaves while another reads its shared memory
}

template <typename W, bool Residual, int U>
__global__ void __launch_bounds__(kThreads *kRcGroups, 1)
k_resample_cluster(W wsrc, RcArgs a)
{
    extern __shared__ __align__(16) unsigned char rc_smem[];
    rc_resample<W, Residual, U>(wsrc, a,
                                *reinterpret_cast<RcShared *>(rc_smem));
}

// CTAs and groups for nt tiles: a tile a CTA up to 16 tiles, then two.
struct RcShape {
    int ctas, groups;
};

inline RcShape rc_shape(int nt)
{
    RcShape s;
    s.groups = nt > kRcMaxCtas ? kRcGroups : 1;
    s.ctas = 1;
    while (s.ctas * s.groups < nt)
        s.ctas *= 2;
    return s;
}

// Launches `k` with one cluster of `shape` per `clusters`.
template <typename K, typename... A>
inline cudaError_t rc_launch(K k, RcShape shape, int clusters,
                             cudaStream_t s, const A &...args)
{
    const size_t smem = rc_smem_bytes(shape.groups);
    cudaError_t e = cudaFuncSetAttribute(
        k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && shape.ctas > 8)
        e = cudaFuncSetAttribute(
            k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess)
        return e;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)(shape.ctas * clusters));
    c.blockDim = dim3((unsigned)(kThreads * shape.groups));
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)shape.ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k, args...);
}

// Whether a resampling of N weights to Nout children (0: N) runs in one
// cluster: its weights and its uniforms must fit in kRcMaxTiles tiles.
inline bool rc_fits(long long N, long long Nout)
{
    const long long n = Nout > N ? Nout : N;
    return resample_ntiles(n) <= kRcMaxTiles;
}

// A resampling: one cluster where it fits, the launch sequence of
// resample.cuh otherwise (and for caller-supplied uniforms).
template <typename W>
inline void launch_resample(int scheme, W wsrc, long long N,
                            const EngineRef &eng, ResampleWorkspace &ws,
                            const double *u_given, long long n_given,
                            bool spine_done, int32_t *rep_out,
                            int32_t *copy_from, cudaStream_t s,
                            bool cfrp = true, long long Nout = 0)
{
    if (u_given != nullptr || !rc_fits(N, Nout) ||
        (W::kExactNorm && !spine_done)) {
        launch_resample_core(scheme, wsrc, N, eng, ws, u_given, n_given,
                             spine_done, rep_out, copy_from, s, false, cfrp,
                             Nout);
        return;
    }
    RcArgs a;
    a.N = N;
    a.nt = resample_ntiles(N);
    a.cfrp = cfrp ? 1 : 0;
    a.spine_done = spine_done ? 1 : 0;
    a.ctl = ws.ctl;
    a.eng = eng;
    a.tile_excl = ws.tile_excl;
    a.u = ws.u;
    a.bins = ws.bins;
    a.rec = ws.ex.rec;
    a.rep_out = rep_out;
    a.copy_from = copy_from;
    const RcShape sh = rc_shape(resample_ntiles(Nout > N ? Nout : N));
    switch (scheme) {
    case VSMC_CUDA_MULTINOMIAL:
        rc_launch(k_resample_cluster<W, false, kRcSorted>, sh, 1, s, wsrc, a);
        break;
    case VSMC_CUDA_RESIDUAL:
        rc_launch(k_resample_cluster<W, true, kRcSorted>, sh, 1, s, wsrc, a);
        break;
    case VSMC_CUDA_STRATIFIED:
        rc_launch(k_resample_cluster<W, false, kRcStrat>, sh, 1, s, wsrc, a);
        break;
    case VSMC_CUDA_SYSTEMATIC:
        rc_launch(k_resample_cluster<W, false, kRcSys>, sh, 1, s, wsrc, a);
        break;
    case VSMC_CUDA_RESIDUAL_STRATIFIED:
        rc_launch(k_resample_cluster<W, true, kRcStrat>, sh, 1, s, wsrc, a);
        break;
    default:
        rc_launch(k_resample_cluster<W, true, kRcSys>, sh, 1, s, wsrc, a);
        break;
    }
}

// Kernels launch_resample issues (for the launch counters).
inline int resample_launch_count(long long N, int scheme, bool exact_norm,
                                 bool approx)
{
    return rc_fits(N, 0)
               ? 1
               : resample_launches(scheme, false, exact_norm, approx);
}

} // namespace vsmc_b200
