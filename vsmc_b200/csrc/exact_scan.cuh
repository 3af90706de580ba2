// exact_scan.cuh -- the reference's sequential cumulative weight, exactly,
// computed in parallel.
//
// internal::inversion (resample/common.hpp:76-79) walks the weights with
// `accw += weight[i]`: S_i = fl(S_{i-1} + w_i), S_{-1} = 0, one rounding
// per step.  A parallel scan rounds differently, so a uniform lying within
// the scan's error of a cumulative weight lands in another slot than the
// reference's (about 10^4 of 2^24 copy_from entries per step with the
// reference's own weights and uniforms).  This file reproduces S_i bit for
// bit for non-negative weights:
//
// * While S_{i-1} and S_i lie in one binade [2^E, 2^(E+1)), both are
//   multiples of u = 2^(E-52), so S_i = S_{i-1} + k_i u with k_i = w_i / u
//   rounded to the nearest integer (a tie would depend on the last bit of
//   S_{i-1}).  Over a run of such "clean" elements the sum is an exact
//   integer sum.
// * An approximate prefix G_i with a proven error bound d decides which
//   elements are clean: the windows G_{i-1} +- d and G_i +- d must lie in
//   one binade.  |S_i - G_i| <= (i + 1) ulp(S_i) / 2 (each rounding of the
//   sequential sum) + the error of G (a relative margin of the weight
//   source); each thread uses one bound for its kItems elements,
//   d = (8 i_last + 256) ulp(2 m) + margin * m, m >= every G and w there.
//   The bound is relative to the thread's own prefixes, so no part of G may be
//   formed by subtracting a later thread's weight from a sum that holds it
//   (block_excl_sum, block_prefix): beside a weight 2^53 times all before it
//   the difference is 0 or off by a binade.
// * A zero weight while the prefix is still 0 leaves S at 0: clean, k = 0.
// * The other ("special") elements -- the first, binade crossings,
//   uncertain binades, ties -- are few (about 40 at N = 2^24): the spine
//   kernel visits them in order with one hardware addition each and jumps
//   over clean runs by their exact integer sums.
//
// Phase A (k_exact_tiles_body, per tile): classify, per-tile integer sums,
// the list of the tile's specials and, per element, a record: the exact
// offset of S_i from the S of the tile's last special before it (or of the
// tile's start), or -1 at a special.  Phase B (k_exact_spine_body, one CTA):
// the exact S at every tile start and at every special.  Phase C (in
// k_invert_body): S_i = base + record, one exact addition, with no weight,
// exp or classification.  A tile with more than kExactCap specials
// (possible only for weights built to create ties) is summed element by
// element in phase B, which writes S_i itself into its records.
#pragma once

#include "smc_common.cuh"

namespace vsmc_b200 {

constexpr int kExactCap = 64;         // specials kept per tile
constexpr int kNoBinade = -100000;    // binade of a special element
constexpr int kExactStage = 1540;     // additions the spine stages: 1024
                                      // specials in 256 tiles (and padding)

struct ExactTile {
    unsigned long long k_total; // sum of the clean elements' k
    int nspec;                  // specials of the tile
    int e_last;                 // binade of the last element (if clean)
};

struct ExactSpecial {
    double w;                     // the weight
    unsigned long long k_before;  // clean k of the tile before it
    int idx;                      // index in the tile
    int e_seg;                    // binade of the clean elements before it
};

// One step of the walk over the specials: the clean run before a special,
// then the special's weight (0 where a run ends without one).
struct ExactStep {
    double seg, w;
};

// Device arrays of the exact scan (part of the resampling workspace).
struct ExactScan {
    ExactTile *tiles;       // ntiles
    ExactSpecial *spec;     // ntiles x kExactCap
    double *s_spec;         // ntiles x kExactCap: exact S at each special
    double *start;          // ntiles + 1: exact S before each tile (0 first)
    double *rec;            // N: per-element record (see above)
    int32_t *kint;          // N: floor(N w) (residual schemes)
    // per tile with specials, by rank (those past the spine's shared stage)
    double *s_out;          // exact S after the tile
    unsigned long long *pk; // clean k before the tile
    int32_t *dirty;         // the tile
    int32_t *eaft;          // binade of the clean tiles after it
};

// Binade of a positive normal double: 2^E <= x < 2^(E+1).
__device__ __forceinline__ int exact_binade(double x)
{
    return ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
}

// 2^e for -1022 <= e <= 1023.
__device__ __forceinline__ double exact_pow2(int e)
{
    return __hiloint2double((e + 1023) << 20, 0);
}

// Binade shared by every value of [g - d, g + d], or kNoBinade.
__device__ __forceinline__ int exact_window(double g, double d)
{
    const double lo = __dadd_rn(g, -d), hi = __dadd_rn(g, d);
    if (!(lo > 0x1p-960))
        return kNoBinade;
    const int e = exact_binade(hi);
    return exact_binade(lo) == e ? e : kNoBinade;
}

// The classification of a thread's R consecutive elements of a tile
// (global index i0 + j): approximate tile start `a`, the thread's exclusive
// prefix `pre` of the tile's weights, the weights `w`; first: pre is 0 only
// when every weight of the tile before the thread's is.  Elements at or past
// N count as clean with k = 0 and the previous element's binade.
template <int R>
struct ExactLocal {
    unsigned long long kloc[R]; // clean k of the thread's elements through j
    int e[R];                   // binades
    unsigned special;           // bit j
    int nsp;
};

template <int R>
__device__ __forceinline__ void
exact_classify(long long i0, long long N, const double (&w)[R], double a,
               double pre, double run, double rel, bool first,
               ExactLocal<R> &x)
{
    // one error bound for the thread's elements (run: their sum).  A
    // negative weight (the sign bits) or one that is not finite (m) leaves
    // every element to the spine.
    int signs = 0;
#pragma unroll
    for (int j = 0; j < R; ++j)
        signs |= __double2hiint(w[j]);
    bool bad = false;
    if (signs < 0) { // (a negative zero is a zero)
#pragma unroll
        for (int j = 0; j < R; ++j)
            bad |= !(w[j] >= 0.0);
    }
    double p = __dadd_rn(pre, run);
    const double m = __dadd_rn(a, p);
    const bool ok = !bad && m > 0x1p-960 && m < 0x1p960;
    double d = 0.0;
    if (ok) {
        const double ulp2 = exact_pow2(exact_binade(m) + 1 - 52);
        const double il = (double)(i0 + R - 1);
        d = __dadd_rn(__dmul_rn(__dadd_rn(8.0 * il, 256.0), ulp2),
                      __dmul_rn(rel, m));
    }
    double gp = __dadd_rn(a, pre);
    unsigned long long kr = 0;
    int nsp = 0;
    unsigned long long (&kloc)[R] = x.kloc;
    x.special = 0;
    // the common case: the windows of the thread's first and last prefix
    // lie in one binade, so every window between them does and each of
    // the thread's elements is clean (unless a tie)
    bool fast = false;
    if (ok && i0 > 0 && i0 + R <= N) {
        const int e0 = exact_window(gp, d);
        if (e0 != kNoBinade && e0 == exact_window(m, d)) {
            const double sc = exact_pow2(52 - e0);
            bool slow = false;
            int over = 0; // a high word outside [2^52, 2^53)
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const double kf = __dmul_rn(w[j], sc);
                const double t = __dadd_rn(kf, 0x1p52);
                over |= __double2hiint(t) ^ 0x43300000;
                slow |= fabs(__dadd_rn(__dadd_rn(t, -0x1p52), -kf)) == 0.5;
                kr += (unsigned long long)(__double_as_longlong(t) -
                                           __double_as_longlong(0x1p52));
                kloc[j] = kr;
                x.e[j] = e0;
            }
            fast = !slow && (over & 0xfff00000) == 0;
        }
    }
    int ep = ok && !fast ? exact_window(gp, d) : kNoBinade;
    p = pre;
    int eprev = kNoBinade;
    if (!fast) {
        kr = 0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const long long i = i0 + j;
            p += w[j];
            const double g = __dadd_rn(a, p);
            const int ec = ok ? exact_window(g, d) : kNoBinade;
            if (i < N) {
                bool sp = true;
                unsigned long long k = 0;
                int e = kNoBinade;
                if (i == 0) {
                    // S_{-1} = 0: the first addition is the hardware's
                } else if (first && gp == 0.0 && w[j] == 0.0) {
                    // a leading zero: every weight before it is 0 (sums of
                    // non-negative weights vanish only so)
                    sp = false;
                } else if (ec != kNoBinade && ec == ep) {
                    // k = w / 2^(e-52) rounded to nearest: adding 2^52 rounds
                    // it to an integer; a tie depends on the sum's last bit
                    const double kf = __dmul_rn(w[j], exact_pow2(52 - ec));
                    if (kf < 0x1p52) {
                        const double t = __dadd_rn(kf, 0x1p52);
                        const double kd = __dadd_rn(t, -0x1p52);
                        if (fabs(__dadd_rn(kd, -kf)) != 0.5) {
                            k = (unsigned long long)(__double_as_longlong(t) -
                                                     __double_as_longlong(0x1p52));
                            e = ec;
                            sp = false;
                        }
                    }
                }
                x.e[j] = e;
                if (sp) {
                    x.special |= 1u << j;
                    ++nsp;
                }
                kr += k;
                eprev = e;
            } else {
                x.e[j] = eprev;
            }
            kloc[j] = kr;
            gp = g;
            ep = ec;
        }
    }
    x.nsp = nsp;
}

// Shared memory of one tile's scan (NW warps).
template <int NW>
struct SmemExactScan {
    unsigned long long k[NW]; // clean k of the warp
    unsigned long long s[NW]; // the warp's clean k at its last special
    int n[NW];                // its specials
    int e[NW];                // binade of its last element
};

// A thread's share of a tile's scan: its element records (the exact offset
// from the last special before it or the tile's start, -1 at a special),
// the specials of the tile before its first element, and the tile's sums.
template <int R>
struct ExactRec {
    double rec[R];
    int rank0, nspec;
    unsigned long long ktile;
};

// Phase A for a tile of NW warps with R elements a thread: one scan of the
// clean k over the group; the last special before a thread is found by
// ballots, so the usual warp without specials pays nothing for them.
// sync() is the group's barrier (called twice); special r goes to
// out.spec(r, ...) and the binade of the tile's last element to out.last.
template <int R, int NW, typename Sync, typename Out>
__device__ __forceinline__ void
exact_scan_tile(long long base, long long i0, long long N,
                const double (&w)[R], double a, double pre, double run,
                double rel, bool first, int lane, int wid,
                SmemExactScan<NW> &sm, Sync sync, Out out, ExactRec<R> &r)
{
    constexpr unsigned kAll = 0xffffffffu;
    ExactLocal<R> x;
    exact_classify(i0, N, w, a, pre, run, rel, first, x);
    const unsigned long long kr = x.kloc[R - 1];
    const unsigned long long ki = warp_incl_scan(kr);
    const unsigned long long ke = ki - kr;
    const int elast = (x.special >> (R - 1)) & 1u ? kNoBinade : x.e[R - 1];
    int e_before = __shfl_up_sync(kAll, elast, 1);
    // specials of the warp: their count before the thread and the warp's
    // clean k at the last of them
    const unsigned any = __ballot_sync(kAll, x.nsp != 0);
    int ne = 0;
    bool has = false;
    unsigned long long kb = 0;
    if (any != 0) {
        unsigned long long kat = 0; // kloc at the thread's last special
#pragma unroll
        for (int j = 0; j < R; ++j)
            if ((x.special >> j) & 1u)
                kat = x.kloc[j];
        const int ni = warp_incl_scan(x.nsp);
        const unsigned before = any & ((1u << lane) - 1u);
        const unsigned long long q =
            __shfl_sync(kAll, ke + kat, 31 - __clz(before | 1u));
        has = before != 0;
        kb = has ? q : 0ull;
        ne = ni - x.nsp;
        if (lane == 31) {
            sm.n[wid] = ni;
            sm.s[wid] = x.nsp ? ke + kat : q;
        }
    } else if (lane == 31) {
        sm.n[wid] = 0;
    }
    if (lane == 31) {
        sm.k[wid] = ki;
        sm.e[wid] = elast;
    }
    sync();
    const unsigned long long wk = lane < NW ? sm.k[lane] : 0ull;
    const int wn = lane < NW ? sm.n[lane] : 0;
    const unsigned long long wki = warp_incl_scan(wk);
    r.ktile = __shfl_sync(kAll, wki, 31);
    const unsigned long long kp = __shfl_sync(kAll, wki - wk, wid);
    const unsigned wany = __ballot_sync(kAll, wn != 0);
    int np = 0;
    unsigned long long kbw = 0; // the tile's clean k at the last special
                                // of the earlier warps
    r.nspec = 0;
    if (wany != 0) {
        const int wni = warp_incl_scan(wn);
        r.nspec = __shfl_sync(kAll, wni, 31);
        np = __shfl_sync(kAll, wni - wn, wid);
        const unsigned before = wany & ((1u << wid) - 1u);
        const unsigned long long at =
            wki - wk + (wn != 0 ? sm.s[lane] : 0ull);
        const unsigned long long q =
            __shfl_sync(kAll, at, 31 - __clz(before | 1u));
        kbw = before != 0 ? q : 0ull;
    }
    if (lane == 0)
        e_before = wid > 0 ? sm.e[wid - 1] : kNoBinade;
    sync(); // sm is free again
    const unsigned long long k0 = kp + ke; // clean k before the thread
    unsigned long long kl = has ? kp + kb : kbw; // ... at the last special
    r.rank0 = np + ne;
    const long long last = min(base + (long long)kTile, N) - 1;
    int rank = r.rank0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        if ((x.special >> j) & 1u) {
            if (rank < kExactCap) {
                ExactSpecial q;
                q.w = w[j];
                q.k_before = k0 + x.kloc[j];
                q.idx = (int)(i0 + j - base);
                q.e_seg = j == 0 ? e_before
                                 : ((x.special >> (j > 0 ? j - 1 : 0)) & 1u
                                        ? kNoBinade
                                        : x.e[j > 0 ? j - 1 : 0]);
                out.spec(rank, q);
            }
            ++rank;
            kl = k0 + x.kloc[j];
            r.rec[j] = -1.0;
        } else {
            const unsigned long long K = k0 + x.kloc[j] - kl;
            r.rec[j] = K == 0 ? 0.0
                              : __dmul_rn((double)K, exact_pow2(x.e[j] - 52));
        }
        if (i0 + j == last)
            out.last((x.special >> j) & 1u ? kNoBinade : x.e[j]);
    }
}

// Phase C: the exact S of a thread's elements from their records, the
// tile's exact start and its specials' exact values sv (ranks below
// kExactCap); an overflow tile's records hold S itself.
__device__ __forceinline__ void
exact_values(const double (&rec)[kItems], int rank0, double start,
             const double *sv, bool overflow, double (&S)[kItems])
{
    int r = rank0 - 1; // rank of the last special before element j
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if (overflow) {
            S[j] = rec[j];
            continue;
        }
        // r < kExactCap holds when the records and the specials come from
        // one classification; the clamp keeps the read in bounds
        if (rec[j] < 0.0) {
            ++r;
            S[j] = sv[min(r, kExactCap - 1)];
        } else {
            const double b = r < 0 ? start : sv[min(r, kExactCap - 1)];
            S[j] = __dadd_rn(b, rec[j]);
        }
    }
}

} // namespace vsmc_b200
