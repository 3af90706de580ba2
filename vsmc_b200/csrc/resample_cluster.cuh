// resample_cluster.cuh -- one resampling of a small filter in one launch.
//
// The pipeline of resample.cuh takes 5 to 14 launches.  For a filter of a
// few tiles each of them holds one or a few CTAs' work and costs 4 to 15 us
// of latency: kernel boundary, control block, global-memory round trips
// between producer and consumer.  Here one thread-block cluster runs the
// whole resampling: each group of kTile / R threads owns one tile and keeps
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
// (the same block scans over the same 256 runs of 8 particles).
//
// Bound: latency (FP64 chains, barriers, dependent shared-memory and L2
// reads); see rc_shape for the split and its measurements.
#pragma once

#include <cooperative_groups.h>
#include <type_traits>

#include "resample_launch.cuh"

namespace vsmc_b200 {

namespace cg = cooperative_groups;

constexpr int kRcStage = 256;   // specials of a scan staged per CTA

// How a resampling draws its U01 sequence.
enum { kRcSorted = 0, kRcStrat = 1, kRcSys = 2 };

// A group: the threads of one tile, R consecutive particles each, with a
// named barrier of its own (barriers 1, 2; 0 is __syncthreads).
template <int R>
struct RcThread {
    static constexpr int TT = kTile / R; // threads of the group
    static constexpr int NW = TT / 32;   // its warps
    int grp, tid, lane, wid;
    __device__ __forceinline__ void sync() const
    {
        asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(TT) : "memory");
    }
};

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
    double sv_w[kExactCap], sv_u[kExactCap]; // (rc_walk_slow) exact S at
                                             // the tile's specials
    double red_d[32];
    unsigned long long red_k[32];
    int red_n[32], red_e[32];
    SmemExactScan<32> scn; // (a group of fewer warps uses its front)
    long long bound[2];
    // engine words, overflow tiles' S, uniforms, rank table in turn
    alignas(16) double buf[kUStage];
};

// The gathered records of one exact scan and its walk: the additions in
// order: each tile's specials, then its clean tail.
struct RcWalk {
    ExactTile t[kRcMaxTiles];
    int off[kRcMaxTiles + 1]; // specials before tile t
    ExactStep step[kRcStage + kRcMaxTiles + 8];
    double S[kRcStage + kRcMaxTiles + 8]; // after each step
    double start[kRcMaxTiles + 1];        // before each tile
    int slow; // overflow tiles, or more specials than staged
};

struct RcShared {
    RcWalk w, u;
    double sums[kRcMaxTiles], usums[kRcMaxTiles];
    double total; // the residuals' approximate sum
    long long NN;
    long long kexcl[kRcMaxTiles + 1];
    int zexcl[kRcMaxTiles + 1], E[kRcMaxTiles];
    double u0, delta;
    int kbits;
    unsigned long long offset;
    double excl[kRcMaxTiles]; // the weights' approximate spine (filters)
    double stats[2];          // M, S1
    int run;                  // the step resamples
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
    ResampleCtl *ctl;
    // given weights: the call's engine position and number of children (0:
    // as many as weights), and where its error and new position go
    unsigned long long offset;
    long long Nout;
    ResampleCtl *out;
    EngineRef eng;
    double *u;        // the U01 sequence and its bins
    int32_t *bins;
    double *rec;      // an overflow tile's weights
    int32_t *rep_out;
    int32_t *copy_from;
};

// Exclusive scan over a group (any association: FP64 sums here feed only
// the exact scan's classification, or are integers), without a subtraction.
template <typename T, int R>
__device__ __forceinline__ T rc_excl_scan(T v, T *sh, const RcThread<R> &th,
                                          T &total)
{
    constexpr int NW = RcThread<R>::NW;
    const T inc = warp_incl_scan(v);
    if (th.lane == 31)
        sh[th.wid] = inc;
    const T mine = warp_excl_of(inc);
    th.sync();
    const T xi = warp_incl_scan(th.lane < NW ? sh[th.lane] : T(0));
    total = __shfl_sync(0xffffffffu, xi, 31);
    const T upto = __shfl_sync(0xffffffffu, xi, th.wid > 0 ? th.wid - 1 : 0);
    th.sync();
    return (th.wid > 0 ? upto : T(0)) + mine;
}

// The plain scan's prefixes of a tile in the launch sequence's association:
// each run of kItems values in order, block_excl_scan over the 256 runs,
// then each run's prefixes in order from its offset.  rec: inclusive.
template <int R>
__device__ __forceinline__ void rc_plain_scan(const double (&w)[R],
                                              const RcThread<R> &th,
                                              RcGroup &g, double (&rec)[R],
                                              double &total)
{
    constexpr int Q = kItems / R; // threads of a run
    const int q = th.tid % Q;
    double run = 0.0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double in = __shfl_up_sync(0xffffffffu, run, 1);
        if (q == k) {
            if (k > 0)
                run = in;
#pragma unroll
            for (int j = 0; j < R; ++j)
                run += w[j];
        }
    }
    double *vr = g.buf; // the runs' sums, then their offsets
    if (q == Q - 1)
        vr[th.tid / Q] = run;
    th.sync();
    double inc = 0.0, v = 0.0;
    if (th.tid < kThreads) {
        v = vr[th.tid];
        inc = warp_incl_scan(v);
        if (th.lane == 31)
            g.red_d[th.wid] = inc;
    }
    th.sync();
    if (th.wid == 0) {
        double s = th.lane < kThreads / 32 ? g.red_d[th.lane] : 0.0;
        s = warp_incl_scan(s);
        if (th.lane < kThreads / 32)
            g.red_d[th.lane] = s;
    }
    th.sync();
    if (th.tid < kThreads) {
        const double wexcl = th.wid > 0 ? g.red_d[th.wid - 1] : 0.0;
        vr[th.tid] = wexcl + inc - v;
    }
    total = g.red_d[kThreads / 32 - 1];
    th.sync();
    double s = vr[th.tid / Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double in = __shfl_up_sync(0xffffffffu, s, 1);
        if (q == k) {
            if (k > 0)
                s = in;
#pragma unroll
            for (int j = 0; j < R; ++j) {
                s += w[j];
                rec[j] = s;
            }
        }
    }
    th.sync(); // vr and red_d are free again
}

// Where a group's scan puts its specials and last binade.
struct RcOut {
    RcScan &sc;
    __device__ __forceinline__ void spec(int r, const ExactSpecial &q) const
    {
        sc.spec[r] = q;
    }
    __device__ __forceinline__ void last(int e) const { sc.tile.e_last = e; }
};

// The scan of the group's tile (weights w, approximate start a and exclusive
// prefix pre): the tile's record and specials into `out`, the thread's
// records into r.
template <int R>
__device__ __forceinline__ void
rc_classify(long long base, long long N, const double (&w)[R], double a,
            double pre, double rel, const RcThread<R> &th, RcGroup &g,
            RcScan &out, double *dump, ExactRec<R> &r)
{
    const long long i0 = base + (long long)th.tid * R;
    double run = 0.0;
#pragma unroll
    for (int j = 0; j < R; ++j)
        run += w[j];
    exact_scan_tile(base, i0, N, w, a, pre, run, rel, true, th.lane, th.wid,
                    reinterpret_cast<SmemExactScan<RcThread<R>::NW> &>(g.scn),
                    [&] { th.sync(); }, RcOut{out}, r);
    if (th.tid == 0) {
        out.tile.k_total = r.ktile;
        out.tile.nspec = r.nspec;
    }
    // a tile with more specials than kept: its values for the walk
    if (r.nspec > kExactCap) {
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (i0 + j < N)
                dump[i0 + j] = w[j];
    }
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
        if (lane == 31)
            k.slow = ov != 0 || in > kRcStage;
    }
}

// The walk's additions: a warp per tile.
template <int B>
__device__ __forceinline__ void rc_gather_specials(cg::cluster_group &cl,
                                                   RcShared &sm, RcWalk &k,
                                                   int nt, int G, int w0)
{
    if (k.slow)
        return;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int wq = (threadIdx.x >> 5) - w0;
    for (int t = wq < 0 ? wq + nw : wq; t < nt; t += nw) {
        const int b = k.off[t], n = k.off[t + 1] - b;
        const ExactTile et = k.t[t];
        const RcGroup *rg = cl.map_shared_rank(&sm.g[t % G], t / G);
        const ExactSpecial *sp = rg->scan[B].spec;
        for (int r = lane; r <= n; r += 32) {
            const unsigned long long kb = r > 0 ? sp[r - 1].k_before : 0ull;
            ExactStep st;
            if (r < n) {
                st.seg = exact_clean(sp[r].k_before - kb, sp[r].e_seg);
                st.w = sp[r].w;
            } else {
                st.seg = exact_clean(et.k_total - kb, et.e_last);
                st.w = 0.0;
            }
            k.step[b + t + r] = st;
        }
    }
}

// Phase B of the exact scan (one thread): the additions in order.
__device__ __forceinline__ void rc_walk(RcWalk &k, int nt)
{
    const int n = k.off[nt] + nt;
    double S = 0.0;
    for (int i = 0; i < n; i += 4) { // (reads past n stay in the array)
        ExactStep q[4];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            q[m] = k.step[i + m];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (i + m < n) {
                S = __dadd_rn(__dadd_rn(S, q[m].seg), q[m].w);
                k.S[i + m] = S;
            }
    }
}

// ... with overflow tiles, summed element by element from `vals` (their S
// goes into the group's buffer), or more specials than staged.
template <int B>
__device__ __noinline__ void rc_walk_slow(cg::cluster_group cl, RcShared &sm,
                                          RcWalk &k, int nt, int G, int own,
                                          const double *vals, long long N)
{
    constexpr bool U = B == kRcU;
    double S = 0.0;
    for (int t = 0; t < nt; ++t) {
        k.start[t] = S;
        const ExactTile et = k.t[t];
        const int mine = t - own;
        const bool keep = mine >= 0 && mine < G;
        if (et.nspec <= kExactCap) {
            const RcGroup *rg = cl.map_shared_rank(&sm.g[t % G], t / G);
            unsigned long long kb = 0;
            for (int r = 0; r < et.nspec; ++r) {
                const ExactSpecial sp = rg->scan[B].spec[r];
                S = __dadd_rn(S, exact_clean(sp.k_before - kb, sp.e_seg));
                S = __dadd_rn(S, sp.w);
                if (keep) {
                    if (U)
                        sm.g[mine].sv_u[r] = S;
                    else
                        sm.g[mine].sv_w[r] = S;
                }
                kb = sp.k_before;
            }
            S = __dadd_rn(S, exact_clean(et.k_total - kb, et.e_last));
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

// The exact S before tile t (t <= the tiles walked).
__device__ __forceinline__ double rc_start(const RcWalk &k, int t)
{
    if (k.slow)
        return k.start[t];
    return t == 0 ? 0.0 : k.S[k.off[t] + t - 1];
}

// The exact S of a thread's elements after the walk.
template <bool U, int R>
__device__ __forceinline__ void rc_values(const RcWalk &k, const RcGroup &g,
                                          int tile, const RcThread<R> &th,
                                          const ExactRec<R> &r, double (&S)[R])
{
    if (k.t[tile].nspec > kExactCap) {
        const double *o = g.buf + (U ? kTile : 0) + th.tid * R;
#pragma unroll
        for (int j = 0; j < R; ++j)
            S[j] = o[j];
        return;
    }
    const double *sv =
        k.slow ? (U ? g.sv_u : g.sv_w) : &k.S[k.off[tile] + tile];
    const double start = rc_start(k, tile);
    int q = r.rank0 - 1; // rank of the last special before element j
#pragma unroll
    for (int j = 0; j < R; ++j) {
        if (r.rec[j] < 0.0) {
            ++q;
            S[j] = sv[min(q, kExactCap - 1)];
        } else {
            S[j] = __dadd_rn(q < 0 ? start : sv[min(q, kExactCap - 1)],
                             r.rec[j]);
        }
    }
}

// Engine words [first, first + count) of the group's tile into its buffer
// (count <= kTile + 2): a Threefry block per thread, shared by the threads
// whose words it holds.  Returns the first word's place; barriers inside.
template <int R>
__device__ __forceinline__ const uint64_t *
rc_words(const EngineRef &eng, unsigned long long first, int count,
         const RcThread<R> &th, RcGroup &g)
{
    uint64_t *q = reinterpret_cast<uint64_t *>(g.buf);
    const unsigned long long b0 = first / 4;
    const int s = (int)(first % 4), nb = (s + count + 3) / 4;
    th.sync(); // (earlier reads of the buffer)
    for (int b = th.tid; b < nb; b += RcThread<R>::TT) {
        const u64x4 x =
            threefry4x64_20(ctr64_add(eng.ctr, b0 + b + 1), eng.key);
#pragma unroll
        for (int l = 0; l < 4; ++l)
            q[4 * b + l] = x.v[l];
    }
    th.sync();
    return q + s;
}

// Sum of the tile sums before tile t (for the classification).
__device__ __forceinline__ double rc_before(const double *sums, int t)
{
    double a = 0.0;
    for (int q = 0; q < t; ++q)
        a += sums[q];
    return a;
}

// R consecutive values of a thread (zero past N).
template <typename T, int R>
__device__ __forceinline__ void rc_load(const T *src, long long i0,
                                        long long N, T (&v)[R])
{
    constexpr int B = R * (int)sizeof(T) < 16 ? R * (int)sizeof(T) : 16;
    typedef typename std::conditional<B == 16, int4, int2>::type V;
    if (i0 + R <= N && (reinterpret_cast<uintptr_t>(src) & (B - 1)) == 0) {
        constexpr int P = B / sizeof(T);
#pragma unroll
        for (int j = 0; j < R / P; ++j) {
            const V q = *reinterpret_cast<const V *>(src + i0 + j * P);
            const T *t = reinterpret_cast<const T *>(&q);
#pragma unroll
            for (int m = 0; m < P; ++m)
                v[j * P + m] = t[m];
        }
    } else {
#pragma unroll
        for (int j = 0; j < R; ++j)
            v[j] = i0 + j < N ? src[i0 + j] : T(0);
    }
}

// R consecutive ints to and from shared memory (R a multiple of 2).
template <int R>
__device__ __forceinline__ void rc_put(int *dst, const int (&v)[R])
{
#pragma unroll
    for (int j = 0; j < R; j += 2)
        *reinterpret_cast<int2 *>(dst + j) = make_int2(v[j], v[j + 1]);
}
template <int R>
__device__ __forceinline__ void rc_get(const int *src, int (&v)[R])
{
#pragma unroll
    for (int j = 0; j < R; j += 2) {
        const int2 q = *reinterpret_cast<const int2 *>(src + j);
        v[j] = q.x;
        v[j + 1] = q.y;
    }
}

// R consecutive ints to a caller's array of any alignment.
template <int R>
__device__ __forceinline__ void rc_store(int32_t *dst, long long i0,
                                         long long N, const int (&v)[R])
{
    if (i0 + R <= N && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
        rc_put<R>(dst + i0, v);
    } else {
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (i0 + j < N)
                dst[i0 + j] = v[j];
    }
}

// One resampling; every thread of the cluster calls it.  A filter's
// weights (kExactNorm, kApprox) read M, S1 and the spine in sm.
template <typename W, bool Residual, int U, int R>
__device__ __forceinline__ void rc_resample(W wsrc, const RcArgs &a,
                                            RcShared &sm)
{
    constexpr bool Sys = U == kRcSys;
    constexpr int TT = RcThread<R>::TT;
    cg::cluster_group cl = cg::this_cluster();
    const int G = (int)blockDim.x / TT;
    const int rank = (int)cl.block_rank();
    RcThread<R> th;
    th.grp = (int)threadIdx.x / TT;
    th.tid = (int)threadIdx.x % TT;
    th.lane = th.tid & 31;
    th.wid = th.tid >> 5;
    const int grp = th.grp, gtid = th.tid, lane = th.lane, wid = th.wid;
    const int own = rank * G;
    const int tile = own + grp;
    const int nt = a.nt;
    const long long N = a.N;
    RcGroup &g = sm.g[grp];
    const bool act = tile < nt;
    const long long base = (long long)tile * kTile;
    const long long i0 = base + (long long)gtid * R;
    constexpr bool Given = std::is_same<W, WeightsGiven>::value;
    const long long Nout = Given && a.Nout > 0 ? a.Nout : N;
    const double Nd = (double)Nout;
    wsrc.prepare();
    if (threadIdx.x == 0) {
        sm.offset = Given ? a.offset : a.ctl->offset;
        if (!Residual) {
            sm.NN = Nout;
            sm.delta = __ddiv_rn(1.0, Nd);
            sm.kbits = bin_kbits(Nout);
            sm.u0 = Sys ? __dmul_rn(canonical_u64(threefry_word(
                                        a.eng.key, a.eng.ctr, sm.offset)),
                                    sm.delta)
                        : 0.0;
        }
        if (rank == 0) {
            a.ctl->words = Sys ? 1 : 0;
            if (Given)
                a.ctl->error = 0;
        }
    }
    __syncthreads();

    // ---- the weights --------------------------------------------------
    double w[R]; // as scanned
    int kk[R];   // floor(N w) (residual)
    ExactRec<R> rw;
    double pre = 0.0, coeff_r = 1.0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        w[j] = 0.0;
        kk[j] = 0;
    }
    if (act) {
        typename W::stage_t x[R];
        rc_load(wsrc.stage_src(), i0, N, x);
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (i0 + j < N)
                w[j] = W::kExactNorm ? wsrc.unnorm_stage(x[j])
                                     : wsrc.from_stage(x[j]);
    }
    if (W::kExactNorm) {
        // the sequential sum of exp(lw - M); its reciprocal normalises
        if (act) {
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < R; ++j)
                run += w[j];
            pre = rc_excl_scan(run, g.red_d, th, total);
            rc_classify(base, N, w,
                        __dmul_rn(sm.excl[tile], wsrc.spine_unnorm()),
                        pre, ExactMargin<W>::rel, th, g, g.scan[kRcA], a.rec,
                        rw);
        }
    }
    // the drawn sequence's first stage, beside the weights' (its length is
    // known unless the scheme is residual)
    double tv[R]; // negated terms
    ExactRec<R> ru;
    double pre_u = 0.0;
    const auto terms = [&]() {
        // log(1 - U_n) / (NN - n), negated, and the tile's sum
        const long long NN = sm.NN;
#pragma unroll
        for (int j = 0; j < R; ++j)
            tv[j] = 0.0;
        if (base < NN) {
            const uint64_t *q = rc_words(
                a.eng, sm.offset + (unsigned long long)base,
                (int)min((long long)kTile, NN - base), th, g);
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const long long n = i0 + j;
                if (n < NN) {
                    const double U1 = canonical_u64(q[gtid * R + j]);
                    tv[j] = -__ddiv_rn(fm::fm_log(__dadd_rn(1.0, -U1)),
                                       (double)(NN - n));
                }
            }
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < R; ++j)
                run += tv[j];
            pre_u = rc_excl_scan(run, g.red_d, th, total);
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
                        ExactMargin<TermsNeg>::rel, th, g,
                        g.scan[kRcU], a.u,
                        ru);
    };
    const auto gather_usums = [&](int nu) {
        if ((int)(threadIdx.x >> 5) == 7 && lane < nu)
            sm.usums[lane] =
                cl.map_shared_rank(&sm.g[lane % G], lane / G)->sum_u;
    };
    // u_n = 1 - exp(lmax_n), its running maximum and the bin index
    const auto sorted_values = [&]() {
        const long long NN = sm.NN;
        if (base >= NN)
            return;
        double S[R];
        rc_values<true>(sm.u, g, tile, th, ru, S);
        const double s0 = rc_start(sm.u, tile);
        const double umax =
            tile > 0 ? __dadd_rn(1.0, -fm::fm_exp(-s0)) : -INFINITY;
        double uv[R];
        double tmax = -INFINITY;
#pragma unroll
        for (int j = 0; j < R; ++j) {
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
        th.sync();
        const double wm = warp_max(lane < wid ? g.red_d[lane] : -INFINITY);
        th.sync();
        exc = fmax(exc, wm);
        double m = fmax(umax, exc);
        const int kb = sm.kbits;
        long long kprev = bin_floor(m, kb);
#pragma unroll
        for (int j = 0; j < R; ++j) {
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
        // (two words more in front: a thread's first value needs the two
        // before it)
        const int lead = base > 0 ? 2 : 0;
        const uint64_t *q = rc_words(
            a.eng, off + (unsigned long long)(base - lead),
            (int)min((long long)kTile, NN - base) + lead, th, g);
        const auto at = [&](long long n) {
            return n >= 0 && n < NN ? strat_u(q[n - base + lead], n, delta)
                                    : -INFINITY;
        };
        double raw[R];
#pragma unroll
        for (int j = 0; j < R; ++j)
            raw[j] = at(i0 + j);
        const double p1 = at(i0 - 1), p2 = at(i0 - 2);
        long long kprev = bin_floor(fmax(p1, p2), kb);
        double rprev = p1;
#pragma unroll
        for (int j = 0; j < R; ++j) {
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
        th.sync(); // the words' buffer is free again
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
            rc_gather_specials<B>(cl, sm, sm.w, nt, G, 0);
        if (wu)
            rc_gather_specials<kRcU>(cl, sm, sm.u, nu, G,
                                     nt % (int)(blockDim.x >> 5));
        __syncthreads();
        if (ww && threadIdx.x == 0) {
            if (sm.w.slow)
                rc_walk_slow<B>(cl, sm, sm.w, nt, G, own, a.rec, N);
            else
                rc_walk(sm.w, nt);
        }
        if (wu && threadIdx.x == 32) {
            if (sm.u.slow)
                rc_walk_slow<kRcU>(cl, sm, sm.u, nu, G, own, a.u, sm.NN);
            else
                rc_walk(sm.u, nu);
        }
        __syncthreads();
        if ((ww && sm.w.slow) || (wu && sm.u.slow))
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
        const double coeff = __ddiv_rn(1.0, rc_start(sm.w, nt));
        pre *= coeff;
#pragma unroll
        for (int j = 0; j < R; ++j)
            w[j] = __dmul_rn(w[j], coeff);
    }
    bool exact = true;
    if (Residual) {
        // r = modf(N w, &k); the tile's sums
        double r[R];
        long long ks = 0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            double k = 0.0;
            r[j] = i0 + j < N ? residual_split(w[j], Nd, k) : 0.0;
            kk[j] = (int32_t)k;
            ks += (long long)k;
        }
        if (act) {
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < R; ++j)
                run += fabs(r[j]);
            if (W::kApprox) {
                // the launch sequence's sum: eight strided elements per
                // thread of 256, warp trees, the warps in order
#pragma unroll
                for (int j = 0; j < R; ++j)
                    g.buf[pad8(gtid * R + j)] = fabs(r[j]);
                th.sync();
                if (gtid < kThreads) {
                    double s = 0.0;
#pragma unroll
                    for (int j = 0; j < kItems; ++j) {
                        const int l = j * kThreads + gtid;
                        if (base + l < N)
                            s += g.buf[pad8(l)];
                    }
                    s = warp_sum(s);
                    if (lane == 0)
                        g.red_d[wid] = s;
                }
                th.sync();
                if (gtid == 0) {
                    double t = 0.0;
                    for (int q = 0; q < kThreads / 32; ++q)
                        t += g.red_d[q];
                    g.sum_w = t;
                }
                th.sync();
            } else {
                pre = rc_excl_scan(run, g.red_d, th, total);
                if (gtid == 0)
                    g.sum_w = total;
            }
            long long kt;
            rc_excl_scan(ks, reinterpret_cast<long long *>(g.red_k), th, kt);
            if (gtid == 0)
                g.ksum = kt;
        }
#pragma unroll
        for (int j = 0; j < R; ++j)
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
                long long NN = Nout - ki;
                if (residual_excess(NN, Nout)) {
                    if (rank == 0)
                        a.ctl->error = VSMC_CUDA_EDEGENERATE;
                    NN = 0;
                }
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
                rc_classify(base, N, w, a0, pre, ExactMargin<W>::rel, th, g,
                            g.scan[kRcB], a.rec, rw);
            cl.sync();
            if (U == kRcSorted) {
                gather_usums(utiles());
                __syncthreads();
            }
            walks(std::integral_constant<int, kRcB>(), true, false);
            coeff_r = __ddiv_rn(1.0, rc_start(sm.w, nt));
            if (act) {
                pre *= coeff_r;
#pragma unroll
                for (int j = 0; j < R; ++j)
                    w[j] = __dmul_rn(w[j], coeff_r);
                rc_classify(base, N, w, a0 * coeff_r, pre,
                            ExactMargin<W>::rel, th, g, g.scan[kRcA], a.rec,
                            rw);
            }
        } else if (W::kApprox) {
            coeff_r = __ddiv_rn(1.0, sm.total);
#pragma unroll
            for (int j = 0; j < R; ++j)
                w[j] = __dmul_rn(w[j], coeff_r);
        }
    } else if (W::kExactNorm) {
        if (act)
            rc_classify(base, N, w,
                        __dmul_rn(sm.excl[tile],
                                  __ddiv_rn(wsrc.spine_unnorm(),
                                            rc_start(sm.w, nt))),
                        pre, ExactMargin<W>::rel, th, g, g.scan[kRcB], a.rec,
                        rw);
    } else if (!W::kApprox) {
        // given weights: tile sums first
        if (act) {
            double run = 0.0, total;
#pragma unroll
            for (int j = 0; j < R; ++j)
                run += w[j];
            pre = rc_excl_scan(run, g.red_d, th, total);
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
                        ExactMargin<W>::rel, th, g, g.scan[kRcA], a.rec, rw);
    }
    if (W::kApprox && exact && act) {
        // the plain scan: inclusive prefixes within the tile, the tile's
        // total in fixed point
        double total;
        rc_plain_scan(w, th, g, rw.rec, total);
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
    double Cx[R];
#pragma unroll
    for (int j = 0; j < R; ++j)
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
                for (int j = 0; j < R; ++j)
                    Cx[j] = __dadd_rn(s0, rw.rec[j]);
            }
        } else if (act) {
            rc_values<false>(sm.w, g, tile, th, rw, Cx);
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
    int rep[R];
    int zl[R]; // rank among the tile's slots without offspring, or -1
    if (act) {
        const auto start = [&](int t) {
            return W::kApprox ? sm.w.start[t] : rc_start(sm.w, t);
        };
        const double sa = exact ? start(tile) : 0.0;
        const double sb = exact ? start(tile + 1) : 0.0;
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
        th.sync();
        const long long lo = g.bound[0];
        const long long hi = max(g.bound[1], lo);
        const bool staged = !Sys && (hi - lo) <= kUStage;
        if (staged) {
            for (int k = gtid; k < (int)(hi - lo); k += TT)
                cp_async8(&sw[k], &u[lo + k]);
            cp_async_commit();
            cp_async_wait_all();
        }
        th.sync();
        const int ilo = (int)lo, ihi = (int)hi, iNN = (int)NN, iN = (int)N;
        const int p0 = (int)i0;
        const int tile_last = (int)min(base + (long long)kTile, N) - 1;
        int cnt[R];
        int pos = -1;
        long long gpos = -1;
#pragma unroll
        for (int j = 0; j < R; ++j) {
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
        for (int j = 1; j < R; ++j)
            cnt[j] = max(cnt[j], cnt[j - 1]);
        int prev = __shfl_up_sync(0xffffffffu, cnt[R - 1], 1);
        if (lane == 31)
            g.red_e[wid] = cnt[R - 1];
        th.sync();
        if (lane == 0)
            prev = wid == 0 ? (tile > 0 ? ilo : 0) : g.red_e[wid - 1];
        int zeros = 0, ksum = 0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
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
        int zloc = rc_excl_scan(zeros, g.red_n, th, ztot);
        int kprefix = 0;
        if (Residual)
            kprefix = (int)sm.kexcl[tile] +
                      rc_excl_scan(ksum, g.red_n, th, ktot);
        if (gtid == 0)
            g.zeros = ztot;
        int sc[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int i = p0 + j;
            kprefix += kk[j];
            const int upto =
                (i >= iN - 1) ? (int)Nout : cnt[j] + kprefix;
            zl[j] = -1;
            if (rep[j] == 0) {
                zl[j] = zloc;
                ++zloc;
            }
            sc[j] = upto - (i + 1) + zloc;
            if (i == tile_last)
                g.sinc_last = sc[j];
        }
        rc_put<R>(g.sinc + gtid * R, sc);
        if (a.rep_out != nullptr)
            rc_store(a.rep_out, i0, N, rep);
    }
    cl.sync();
    // the engine position (the words are final)
    if (rank == 0 && threadIdx.x == 0) {
        const unsigned long long off =
            sm.offset + *(volatile unsigned long long *)&a.ctl->words;
        a.ctl->offset = off;
        if (Given) {
            a.out->offset = off;
            a.out->error = *(volatile int *)&a.ctl->error;
        }
    }
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
            int m[R];
#pragma unroll
            for (int j = 0; j < R; ++j)
                m[j] = -1;
            rc_put<R>(tab + gtid * R, m);
            th.sync();
            // parent p owns the ranks [sinc(p - 1), sinc(p)): it marks the
            // first of them that falls in the window
            int prev_top = INT_MIN;
            for (int pt = tf; pt <= tl; ++pt) {
                const long long pb = (long long)pt * kTile;
                const int len = (int)min((long long)kTile, N - pb);
                const int zoff = sm.zexcl[pt];
                const RcGroup *rg = cl.map_shared_rank(&sm.g[pt % G], pt / G);
                int v[R];
                rc_get<R>(rg->sinc + gtid * R, v);
                int before =
                    gtid > 0 ? rg->sinc[gtid * R - 1] + zoff : prev_top;
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const int l = gtid * R + j;
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
            th.sync();
            // parents increase with the rank: the running maximum of the
            // marks is each rank's parent
            rc_get<R>(tab + gtid * R, m);
#pragma unroll
            for (int j = 1; j < R; ++j)
                m[j] = max(m[j], m[j - 1]);
            int in = m[R - 1];
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
            th.sync();
            ex = max(ex, __reduce_max_sync(0xffffffffu,
                                           lane < wid ? g.red_n[lane] : -1));
#pragma unroll
            for (int j = 0; j < R; ++j)
                m[j] = max(m[j], ex);
            rc_put<R>(tab + gtid * R, m);
            th.sync();
        }
        int cf[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            cf[j] = (int)i0 + j;
            if (i0 + j < N && zl[j] >= 0) {
                const int p = zl[j] < min(z, top) ? tab[zl[j]] : -1;
                if (p >= 0)
                    cf[j] = p;
                else // no parent found: replication != N
                    atomicExch(&a.ctl->error, (int)VSMC_CUDA_EDEGENERATE);
            }
        }
        rc_store(a.copy_from, i0, N, cf);
    }
    cl.sync(); // no CTA leaves while another reads its shared memory
    if (Given && rank == 0 && threadIdx.x == 0)
        a.out->error = *(volatile int *)&a.ctl->error;
}

template <typename W, bool Residual, int U, int R>
__global__ void __launch_bounds__(R == 8 ? 512 : kTile / R, 1)
k_resample_cluster(W wsrc, RcArgs a)
{
    extern __shared__ __align__(16) unsigned char rc_smem[];
    rc_resample<W, Residual, U, R>(wsrc, a,
                                   *reinterpret_cast<RcShared *>(rc_smem));
}

// k_cv_finalize_body for at most 32 tiles, by one warp (lane t holds tile
// t, as thread t does there): every CTA of a cluster computes the step's
// maximum, sums and decision, CTA 0 writes them.  Leaves M, S1, the spine
// and the decision in sm.
__device__ __forceinline__ void rc_finalize(const FinalizeArgs &a,
                                            RcShared &sm, bool writer)
{
    const int lane = threadIdx.x & 31;
    FilterCtl *c = a.ctl;
    int c_res = 0;
    long long c_mdone = 0;
    double c_s1 = 0.0, c_logz = 0.0;
    double ax0 = 0.0, ay0 = 0.0, ax1 = 0.0, ay1 = 0.0;
    if (writer && lane == 0) {
        c_res = c->resampled;
        c_mdone = c->monitor_done;
        c_s1 = c->s1;
        c_logz = c->logz;
        if (a.anchored) {
            if (!a.init) {
                ax0 = a.obs_x[a.t - 1];
                ay0 = a.obs_y[a.t - 1];
            }
            ax1 = a.obs_x[a.t];
            ay1 = a.obs_y[a.t];
        }
    }
    const int rflag =
        a.replay_flags != nullptr ? a.replay_flags[a.t] : 0;
    TileStats ts;
    ts.m = -INFINITY;
    ts.s1 = ts.s2 = ts.sx = ts.sy = ts.gx = ts.gy = 0.0;
    if (lane < a.ntiles)
        ts = a.ts[lane];
    double M = (ts.m != ts.m || ts.s1 != ts.s1) ? NAN : ts.m;
    for (int o = 16; o > 0; o >>= 1) {
        const double q = __shfl_xor_sync(0xffffffffu, M, o);
        M = (q != q || M != M) ? NAN : fmax(M, q);
    }
    const double f = ts.m == -INFINITY ? 0.0 : fm::fm_exp(ts.m - M);
    const double share = __dmul_rn(ts.s1, f);
    const double S1 = warp_sum(share);
    const double S2 = warp_sum(__dmul_rn(__dmul_rn(ts.s2, f), f));
    const double sx = warp_sum(__dmul_rn(ts.sx, f));
    const double sy = warp_sum(__dmul_rn(ts.sy, f));
    const double gx = warp_sum(ts.gx), gy = warp_sum(ts.gy);
    const double Nd = (double)a.N;
    const bool bad = !(M > -INFINITY && M < INFINITY && S1 > 0.0 &&
                       S1 < INFINITY && S2 > 0.0 && S2 < INFINITY);
    const double ess = bad ? NAN : S1 * S1 / S2;
    const int own = bad ? 0 : ess < a.threshold * Nd;
    // the step's own decision resamples unless the step follows a recorded
    // ancestry without comparing
    const int run = a.replay_flags == nullptr || a.compare ? own : 0;
    const int res = a.replay_flags != nullptr ? rflag != 0 : own;
    // the spine of the normalised shares, for the classification
    const double sh = share * __ddiv_rn(1.0, S1);
    const double excl = warp_excl_of(warp_incl_scan(sh));
    sm.excl[lane] = excl;
    if (lane != 0)
        return;
    sm.stats[0] = M;
    sm.stats[1] = S1;
    sm.run = run;
    if (!writer)
        return;
    // monitor of the previous step, gathered by this move
    if (!a.init && c_res && c_mdone != a.t - 1) {
        a.hist_mean_x[a.t - 1] = ax0 + gx / Nd;
        a.hist_mean_y[a.t - 1] = ay0 + gy / Nd;
        c->monitor_done = a.t - 1;
    }
    const double s1prev = (a.init || c_res) ? Nd : c_s1;
    const double dz = bad ? NAN : M + log(S1) - log(s1prev);
    if (bad)
        c->error = VSMC_CUDA_EDEGENERATE;
    a.hist_ess[a.t] = ess;
    a.hist_resampled[a.t] = res;
    a.hist_logz_inc[a.t] = dz;
    c->logz = c_logz + dz;
    c->lw_max = M;
    c->s1 = S1;
    c->s2 = S2;
    c->ess = ess;
    c->resampled = res;
    if (!res) {
        a.hist_mean_x[a.t] = ax1 + sx / S1;
        a.hist_mean_y[a.t] = ay1 + sy / S1;
    }
    a.rctl->active = run;
}

// A step's finalisation and resampling.
template <typename W, bool Residual, int U, int R>
__global__ void __launch_bounds__(R == 8 ? 512 : kTile / R, 1)
k_finish_cluster(FinalizeArgs fa, W wsrc, RcArgs a)
{
    extern __shared__ __align__(16) unsigned char rc_smem[];
    RcShared &sm = *reinterpret_cast<RcShared *>(rc_smem);
    pdl_wait();
    pdl_launch(); // the next move draws its normals meanwhile
    if (threadIdx.x < 32)
        rc_finalize(fa, sm, cg::this_cluster().block_rank() == 0);
    __syncthreads();
    if (!sm.run)
        return; // (the whole cluster: every CTA takes the same decision)
    wsrc.stats = sm.stats;
    rc_resample<W, Residual, U, R>(wsrc, a, sm);
}

// The cluster of nt tiles: up to 16 a CTA of 1024 threads each (two
// particles a thread), above two tiles a CTA of 512 threads (eight).  The
// serial chain over a thread's particles is what a tile waits for, so few
// particles a thread are better as long as an SM's threads suffice: two
// tiles a CTA leave 1024 threads for 4096 particles, and there the fewer
// registers of 1024-thread CTAs cost more than the shorter chain gives.
// FP64 Multinomial filter, us a step at N = 1000 / 32768 / 65536 on one
// B200: launch sequence 93.8 / 112.8 / 113; this cluster with 256 threads a
// tile 62.7 / 83.0 / 89.9; as it is 48.0 / 65.1 / 82.6; with the
// finalisation in the same kernel 37.5 / 46.0 / 63.8; launched early 31.7 /
// - / 57.2.
struct RcShape {
    int ctas, groups, r;
};

inline RcShape rc_shape(int nt)
{
    RcShape s;
    s.groups = nt > kRcMaxCtas ? kRcGroups : 1;
    s.r = nt > kRcMaxCtas ? 8 : 2;
    s.ctas = 1;
    while (s.ctas * s.groups < nt)
        s.ctas *= 2;
    return s;
}

// Launches `k` as one cluster of `shape`; `early`: before the stream's
// previous kernel has ended (k waits itself).  False: no room for the
// cluster, nothing launched.
template <typename K, typename... A>
inline bool rc_launch(K k, RcShape shape, bool early, cudaStream_t s,
                      const A &...args)
{
    const size_t smem = rc_smem_bytes(shape.groups);
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    if (shape.ctas > 8)
        cudaFuncSetAttribute(
            k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)shape.ctas);
    c.blockDim = dim3((unsigned)(kTile / shape.r * shape.groups));
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)shape.ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = early ? 2 : 1;
    if (!cluster_room(k, c))
        return false;
    cudaLaunchKernelEx(&c, k, args...);
    return true;
}

// The scheme's instance: f(residual, sequence) with compile-time constants.
template <typename F>
inline void rc_scheme(int scheme, F f)
{
    typedef std::integral_constant<int, kRcSorted> Sorted;
    typedef std::integral_constant<int, kRcStrat> Strat;
    typedef std::integral_constant<int, kRcSys> Syst;
    switch (scheme) {
    case VSMC_CUDA_MULTINOMIAL:
        f(std::false_type(), Sorted());
        break;
    case VSMC_CUDA_RESIDUAL:
        f(std::true_type(), Sorted());
        break;
    case VSMC_CUDA_STRATIFIED:
        f(std::false_type(), Strat());
        break;
    case VSMC_CUDA_SYSTEMATIC:
        f(std::false_type(), Syst());
        break;
    case VSMC_CUDA_RESIDUAL_STRATIFIED:
        f(std::true_type(), Strat());
        break;
    default:
        f(std::true_type(), Syst());
        break;
    }
}

inline RcArgs rc_args(long long N, const EngineRef &eng,
                      const ResampleWorkspace &ws, int32_t *rep_out,
                      int32_t *copy_from, bool cfrp)
{
    RcArgs a;
    a.N = N;
    a.nt = resample_ntiles(N);
    a.cfrp = cfrp ? 1 : 0;
    a.ctl = ws.ctl;
    a.offset = 0;
    a.Nout = 0;
    a.out = ws.ctl;
    a.eng = eng;
    a.u = ws.u;
    a.bins = ws.bins;
    a.rec = ws.ex.rec;
    a.rep_out = rep_out;
    a.copy_from = copy_from;
    return a;
}

template <typename W>
bool launch_cluster_finish(int scheme, const FinalizeArgs &fa, const W &w,
                           const ResampleWorkspace &ws, int32_t *copy_from,
                           cudaStream_t s)
{
    bool done = false;
    const RcArgs a = rc_args(fa.N, fa.eng, ws, nullptr, copy_from, true);
    const RcShape sh = rc_shape(fa.ntiles);
    rc_scheme(scheme, [&](auto res, auto u) {
        constexpr bool Re = decltype(res)::value;
        constexpr int U = decltype(u)::value;
        if (sh.r == 8)
            done = rc_launch(k_finish_cluster<W, Re, U, 8>, sh, true, s, fa, w,
                             a);
        else
            done = rc_launch(k_finish_cluster<W, Re, U, 2>, sh, true, s, fa, w,
                             a);
    });
    return done;
}

} // namespace vsmc_b200
