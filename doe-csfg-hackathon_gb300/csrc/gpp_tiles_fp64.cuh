// gpp_tiles_fp64.cuh -- FP64 tile bodies of the GPP sigma kernels, shared by
// the one-state kernels (gpp_fp64.cu) and the persistent batched kernels.
//
// Algorithm (reference: noflagOCC_solver gppComplex_seq.cpp:131-150,
// flagOCC_solver :107-128, ssxt_scht_solver :16-63, driver :335-383).
// The unoccupied term is regrouped, exactly in real arithmetic, as
//
//   mygpvar1 aqsn (delw I_eps) = conj(aqsm[n1,igp]) * A * conj(wdiff) / |wdiff|^2
//   A = aqsn[n1,ig] * (wtilde[igp,ig] * I_eps[igp,ig]),  wdiff = wx - wtilde
//
// so conj(aqsm) leaves the ig sum (applied once per (n1,igp) in the block
// epilogue) and A is shared by all frequencies.  Per term the FP64 pipe then
// does 9 instructions: wdiff.re (DADD), |wdiff|^2 (DFMA), the reciprocal (3
// DFMA after a seed from the multi-function unit), A*conj(wdiff) (2 DFMA with
// the iw-independent products hoisted) and the accumulation (2 DFMA).
//
// Work decomposition: a tile is RG local G' rows x RN bands x NWC
// frequencies and all ncouls columns; the block's threads stride over ig, so
// every global load is a coalesced 16-byte double2 (ld.global.nc) and each
// loaded element is reused RN*NWC (rows) or RG*NWC (bands) times from
// registers.  Partial sums: per-thread registers -> warp shuffle tree ->
// shared-memory tree across warps -> one complex per tile and frequency in
// the workspace, summed over tiles in a fixed order by the reduction kernel.
#pragma once

#include <type_traits>

#include "gpp_internal.cuh"

namespace gpp {

// One unoccupied-band tile in FP64: rows row_tile*RG.., bands
// band_begin + band_tile*RN.., frequencies iw_chunk*NWC..; `tile` is the
// tile's index inside this launch's block-partial segment.  red/S are
// shared-memory scratch of (THREADS/32)*K and K doubles, K = RN*RG*NWC*2.
template <int RN, int RG, int NWC, int THREADS>
__device__ __forceinline__ void noflag_fp64_tile(const Problem &p, const Partials &part,
                                                 int band_begin, int band_end, int row_tile,
                                                 int band_tile, int iw_chunk, long long tile,
                                                 double *red, double *S) {
    constexpr int K = RN * RG * NWC * 2;
    const int row0 = row_tile * RG;
    const int band0 = band_begin + band_tile * RN;
    const int iw0 = iw_chunk * NWC;
    const int nc = p.nc;

    const double2 *wrow[RG];
    const double2 *erow[RG];
#pragma unroll
    for (int g = 0; g < RG; ++g) {
        const int r = min(row0 + g, p.ng - 1);
        wrow[g] = p.wt + (size_t)r * nc;
        erow[g] = p.ieps + (size_t)r * nc;
    }
    const double2 *nrow[RN];
    double wx[RN][NWC];
#pragma unroll
    for (int n = 0; n < RN; ++n) {
        const int b = min(band0 + n, band_end - 1);
        nrow[n] = p.aqsn + (size_t)b * nc;
#pragma unroll
        for (int w = 0; w < NWC; ++w)
            wx[n][w] = __ldg(p.wx + (size_t)b * p.wx_stride + min(iw0 + w, p.nw - 1));
    }

    double2 acc[RN][RG][NWC];
#pragma unroll
    for (int n = 0; n < RN; ++n)
#pragma unroll
        for (int g = 0; g < RG; ++g)
#pragma unroll
            for (int w = 0; w < NWC; ++w) acc[n][g][w] = make_double2(0.0, 0.0);

    for (int ig = threadIdx.x; ig < nc; ig += THREADS) {
        double2 Q[RG];
        double wtr[RG], wti[RG], wti2[RG];
#pragma unroll
        for (int g = 0; g < RG; ++g) {
            const double2 wt = __ldg(wrow[g] + ig);
            const double2 ie = __ldg(erow[g] + ig);
            Q[g] = cmul(wt, ie);
            wtr[g] = wt.x;
            wti[g] = wt.y;
            wti2[g] = wt.y * wt.y;
        }
#pragma unroll
        for (int n = 0; n < RN; ++n) {
            const double2 a = __ldg(nrow[n] + ig);
#pragma unroll
            for (int g = 0; g < RG; ++g) {
                const double2 A = cmul(a, Q[g]);
                const double ayw = A.y * wti[g];
                const double axw = A.x * wti[g];
#pragma unroll
                for (int w = 0; w < NWC; ++w) {
                    const double wr = wx[n][w] - wtr[g];   // Re(wdiff); Im(wdiff) = -wti
                    const double d = fma(wr, wr, wti2[g]); // |wdiff|^2
                    const double r = rcp_fp64(d);
                    const double tx = fma(A.x, wr, -ayw);  // A * conj(wdiff)
                    const double ty = fma(A.y, wr, axw);
                    acc[n][g][w].x = fma(r, tx, acc[n][g][w].x);
                    acc[n][g][w].y = fma(r, ty, acc[n][g][w].y);
                }
            }
        }
    }

    double v[K];
#pragma unroll
    for (int n = 0; n < RN; ++n)
#pragma unroll
        for (int g = 0; g < RG; ++g)
#pragma unroll
            for (int w = 0; w < NWC; ++w) {
                const int k = ((n * RG + g) * NWC + w) * 2;
                v[k] = acc[n][g][w].x;
                v[k + 1] = acc[n][g][w].y;
            }
    block_reduce<K, THREADS>(v, red, S);

    noflag_epilogue<RN, RG, NWC>(p, part, S, row0, band0, band_end, iw0, tile, row_tile);
}

// Epilogue of an occupied-band tile: S holds, per (row g, frequency w), the
// ig sums of aqsn*sch and aqsn*ssx as S[(g*NWC + w)*4 + {0,1 | 2,3}].  Weight
// by conj(aqsm[band,igp]) (the matngmatmgp factor) and by 0.5 vcoul[igp]
// (achtemp) or occ vcoul[igp] (asxtemp), gppComplex_seq.cpp:359-363,378-381;
// threads 0..NWC-1 write achtemp partials, NWC..2NWC-1 asxtemp partials and
// thread 64 the iw = 2 column of acht_n1_loc.
template <int RG, int NWC>
__device__ __forceinline__ void flag_epilogue(const Problem &p, const Partials &part,
                                              const double *S, int row0, int band, int iw0,
                                              long long tile, int row_tile) {
    const int nc = p.nc;
    const int t = threadIdx.x;
    // t < NWC: achtemp partial; NWC <= t < 2 NWC: asxtemp partial; t == 64: n1 column.
    const bool do_ach = t < NWC, do_asx = t >= NWC && t < 2 * NWC, do_n1 = part.n1 && t == 64;
    if (do_ach || do_asx || do_n1) {
        const int w = do_ach ? t : (do_asx ? t - NWC : 2 - iw0);
        if (w >= 0 && w < NWC && iw0 + w < p.nw) {
            double2 tot = make_double2(0.0, 0.0);
#pragma unroll
            for (int g = 0; g < RG; ++g) {
                const int row = row0 + g;
                if (row >= p.ng) continue;
                const int igp = resolve_igp(p, row, part.err);
                if (igp < 0) continue;
                const double2 m = __ldg(p.aqsm + (size_t)band * nc + igp);
                const int k = (g * NWC + w) * 4 + (do_asx ? 2 : 0);
                const double2 s =
                    cmul_rn(make_double2(m.x, -m.y), make_double2(S[k], S[k + 1]));
                const double v_igp = __ldg(p.vcoul + igp);
                const double2 t = do_asx ? cscale_rn(s, __dmul_rn(p.occ, v_igp))
                                         : cscale_rn(cscale_rn(s, 0.5), v_igp);
                tot = make_double2(__dadd_rn(tot.x, t.x), __dadd_rn(tot.y, t.y));
            }
            if (do_ach)
                part.ach[(long long)(iw0 + w) * part.ach_seg + part.ach_tile0 + tile] = tot;
            else if (do_asx)
                part.asx[(long long)(iw0 + w) * part.asx_seg + tile] = tot;
            else
                part.n1[(long long)band * part.n1_seg + row_tile] = tot;
        }
    }
}

// a > t and a < t for a, t >= 0 (t finite), on the bits: the order of the bit
// patterns is that of the values, and NaN (any sign) compares false as it
// does in FP64.  Integer compares keep the tests off the FP64 pipe.
__device__ __forceinline__ bool pos_gt(double a, double t) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(a);
    return u > (unsigned long long)__double_as_longlong(t) && u <= 0x7FF0000000000000ull;
}
__device__ __forceinline__ bool pos_lt(double a, double t) {
    return (unsigned long long)__double_as_longlong(a) <
           (unsigned long long)__double_as_longlong(t);
}

// What an occupied-band tile keeps per frequency (uniform over the block):
// c = wx^2, and how the branch-A sum of aqsn Omega2 is formed.  Away from
// small wx nearly every term is branch A and `most` is set: the tile sums
// aqsn Omega2 once for all frequencies, over the columns with
// |wtilde|^2 <= flag_bound (none of which any frequency's cutoff takes), and
// each frequency adds or takes off only the terms where its own set differs.
// What is taken off lies near the frequency (|wtilde| about |wx|), so the
// difference loses nothing; with a small wx the 1/wx^2 scale would enlarge
// its rounding, and those frequencies add their terms one by one.  Where wx^2 or
// its inverse would leave FP64's range, or float's for the mixed tile, `plain`
// is not set: the terms are then summed with 1/wx^2 in branch A and nothing in
// branch B.
struct FlagFreq {
    double wx, c;
    bool most, cut, plain;
};
// x with its sign bit flipped where `neg` is set (no FP64 instruction).
__device__ __forceinline__ double flip(double x, bool neg) {
    return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}
template <int SEM>
__device__ __forceinline__ FlagFreq flag_freq(double wx) {
    FlagFreq f;
    f.wx = wx;
    f.c = __dmul_rn(wx, wx);
    f.cut = SEM == kSemComplexSeq && wx < 0.0;
    f.plain = fabs(wx) >= 1e-12 && fabs(wx) < 1e15;
    f.most = f.plain && fabs(wx) >= 1.0;
    return f;
}
constexpr double kFlagNoBound = 1.7976931348623157e308;  // the largest double
// The smallest |wtilde|^2 at which a frequency's branch-A cutoff starts.
__device__ __forceinline__ double flag_bound(double bound, const FlagFreq &f) {
    const double t = __dmul_rn(4.0, f.c);
    return f.cut && t < bound ? t : bound;
}
// 1/wx^2 of branch A as the reference forms it (wx^2 / pow(wx^2, 2),
// gppComplex_seq.cpp:38-41), and what the sum y of a frequency's terms times
// wx^2 (not plain: of its terms) stands for; no terms give 0 whatever wx is.
__device__ __forceinline__ double flag_inverse(double c) { return c / (c * c); }
__device__ __forceinline__ double flag_ssx_scale(const FlagFreq &f, double y) {
    return !f.plain || y == 0.0 ? y : __dmul_rn(y, flag_inverse(f.c));
}

// ssxt_scht_solver (gppComplex_seq.cpp:16-63) for one (row, column,
// frequency) and NB bands, accumulated as acc_s += aqsn sch and
// y += wx^2 aqsn ssx (where f.plain; the conj(aqsm) factor of matngmatmgp and 1/wx^2 are
// applied to the sums).  In exact arithmetic, with Q = wtilde I_eps and
// A = aqsn Q:
//   branch A (|wdiff|^2 > limittwo, |delw|^2 = |wtilde|^2 / |wdiff|^2 < limitone):
//     aqsn sch = A conj(wdiff) / |wdiff|^2,  wx^2 aqsn ssx = aqsn Omega2 = A wtilde;
//   branch B (|delw|^2 > to1): sch = 0 and, as Omega2 = wtilde^2 I_eps and
//     cden = 4 wtilde^2 (0.5 + delw), ssx = -Omega2 delw / cden
//     = -Q / (2 (wx + wtilde));
//   the cutoff |ssx| > 4 |I_eps| is |wtilde|^2 > 4 wx^2 in branch A and
//     |wtilde|^2 > 64 |wx + wtilde|^2 in branch B.
// Bound by the FP64 pipe: 28 instructions per (row, column, frequency) of two
// bands (6 shared, 4 per band, the rest per column; ncu), where evaluating
// delw, Omega2, cden and the products as the reference does took 66.  819 x
// 16384, two bands, 3 frequencies: 2.3 ms, the pipe 87% busy.  Every rounding
// is explicit, so a band gives the same bits alone and beside another one.
// in_all: whether the sum over all columns holds this one.  PLAIN: every
// frequency of the tile is known to be plain (tested term by term, the FP64 drop-in
// call of 512 bands x 1638 x 32768 took 19.8 ms; 19.3 with this).
struct FlagSolve {
    double wr, rden, delwr;  // Re(wdiff) (Im(wdiff) = -Im(wtilde)), 1 / |wdiff|^2, |delw|^2
    bool in_a;
};
__device__ __forceinline__ FlagSolve flag_solve(const FlagFreq &f, double2 wt, double wti2,
                                                double awt2) {
    FlagSolve s;
    s.wr = __dsub_rn(f.wx, wt.x);
    const double d = __fma_rn(s.wr, s.wr, wti2);
    s.rden = rcp_fp64(d);
    s.delwr = __dmul_rn(awt2, s.rden);
    s.in_a = pos_gt(d, kLimitTwo) && pos_lt(s.delwr, kLimitOne);
    return s;
}
// acc += A conj(wdiff) / |wdiff|^2, with Aw = A Im(wtilde).
__device__ __forceinline__ void flag_sch(const FlagSolve &s, double2 A, double2 Aw, double2 &acc) {
    acc.x = __fma_rn(s.rden, __fma_rn(A.x, s.wr, -Aw.y), acc.x);
    acc.y = __fma_rn(s.rden, __fma_rn(A.y, s.wr, Aw.x), acc.y);
}
template <int NB, bool PLAIN = false>
__device__ __forceinline__ void flag_ssx(const FlagFreq &f, const FlagSolve &s, bool in_all,
                                         double2 wt, double wti2, double awt2,
                                         const double2 (&A)[NB], const double2 (&Aw)[NB],
                                         const double2 (&B)[NB], double2 (&y)[NB]) {
    const bool inc = s.in_a && !(f.cut && pos_gt(awt2, __dmul_rn(4.0, f.c)));
    const bool base = f.most && in_all;
    if (!PLAIN && inc && !f.plain) {
        const double inv = flag_inverse(f.c);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            y[b].x = __fma_rn(B[b].x, inv, y[b].x);
            y[b].y = __fma_rn(B[b].y, inv, y[b].y);
        }
    } else if (inc != base) {  // a branch-A term to add, or one to take off the sum over all columns
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            y[b].x = __dadd_rn(y[b].x, flip(B[b].x, base));
            y[b].y = __dadd_rn(y[b].y, flip(B[b].y, base));
        }
    }
    if (!s.in_a && pos_gt(s.delwr, kTo1)) {
        const double sr = __dadd_rn(f.wx, wt.x);  // wx + wtilde = (sr, Im(wtilde))
        const double rs = rcp_fp64(__fma_rn(sr, sr, wti2));
        if (!(f.cut && pos_gt(__dmul_rn(awt2, rs), 64.0))) {
            const double m = __dmul_rn(__dmul_rn(-0.5, PLAIN || f.plain ? f.c : 1.0), rs);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                y[b].x = __fma_rn(m, __fma_rn(A[b].x, sr, Aw[b].y), y[b].x);
                y[b].y = __fma_rn(m, __fma_rn(A[b].y, sr, -Aw[b].x), y[b].y);
            }
        }
    }
}

template <int NB, bool PLAIN = false>
__device__ __forceinline__ void flag_term(const FlagFreq &f, bool in_all, double2 wt, double wti2,
                                          double awt2, const double2 (&A)[NB], const double2 (&Aw)[NB],
                                          const double2 (&B)[NB], double2 (&acc_s)[NB],
                                          double2 (&y)[NB]) {
    const FlagSolve s = flag_solve(f, wt, wti2, awt2);
    if (s.in_a) {
#pragma unroll
        for (int b = 0; b < NB; ++b) flag_sch(s, A[b], Aw[b], acc_s[b]);
    }
    flag_ssx<NB, PLAIN>(f, s, in_all, wt, wti2, awt2, A, Aw, B, y);
}

// The products of one (row, column) that its frequencies share: A = aqsn Q,
// Aw = A Im(wtilde) and B = A wtilde = aqsn Omega2; wti2 = Im(wtilde)^2 and
// awt2 = |wtilde|^2.
template <int NB>
__device__ __forceinline__ void flag_products(double2 wt, double2 ie, const double2 (&a)[NB],
                                              double &wti2, double &awt2, double2 (&A)[NB],
                                              double2 (&Aw)[NB], double2 (&B)[NB]) {
    const double2 Q = cmul_rn(wt, ie);
    wti2 = __dmul_rn(wt.y, wt.y);
    awt2 = __fma_rn(wt.x, wt.x, wti2);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        A[b] = cmul_rn(a[b], Q);
        Aw[b] = cscale_rn(A[b], wt.y);
        B[b] = make_double2(__fma_rn(A[b].x, wt.x, -Aw[b].y), __fma_rn(A[b].y, wt.x, Aw[b].x));
    }
}

// One occupied-band tile in FP64: rows row_tile*RG.., bands [band0,
// band0 + NB), frequencies iw_chunk*NWC..; red/S are shared scratch of
// (THREADS/32)*K and K doubles, K = NB*RG*NWC*4.  NB > 1 is for
// band-independent frequencies (wx_stride == 0): |wdiff|^2, its reciprocal
// and the branch are formed once for all NB bands; per band the operations,
// their order and the reduction tree are those of NB = 1, and so the bits.
// Bands past nv (a ragged last group) are computed on a clamped band and not
// written.
template <int RG, int NWC, int NB, int THREADS, int SEM>
__device__ __forceinline__ void flag_fp64_tile(const Problem &p, const Partials &part,
                                               int row_tile, int band0, int iw_chunk,
                                               int row_tiles, double *red, double *S) {
    constexpr int KB = RG * NWC * 4, K = NB * KB;
    const int row0 = row_tile * RG;
    const int iw0 = iw_chunk * NWC;
    const int nc = p.nc;

    const double2 *wrow[RG];
    const double2 *erow[RG];
#pragma unroll
    for (int g = 0; g < RG; ++g) {
        const int r = min(row0 + g, p.ng - 1);
        wrow[g] = p.wt + (size_t)r * nc;
        erow[g] = p.ieps + (size_t)r * nc;
    }
    const double2 *nrow[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) nrow[b] = p.aqsn + (size_t)min(band0 + b, p.nv - 1) * nc;
    FlagFreq f[NWC];
    double bound = kFlagNoBound;
    bool any_most = false, all_plain = true;
#pragma unroll
    for (int w = 0; w < NWC; ++w) {
        f[w] = flag_freq<SEM>(__ldg(p.wx + (size_t)band0 * p.wx_stride + min(iw0 + w, p.nw - 1)));
        bound = flag_bound(bound, f[w]);
        any_most |= f[w].most;
        all_plain &= f[w].plain;
    }

    double2 acc_s[RG][NWC][NB], y[RG][NWC][NB], all[RG][NB];
#pragma unroll
    for (int g = 0; g < RG; ++g)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            all[g][b] = make_double2(0.0, 0.0);
#pragma unroll
            for (int w = 0; w < NWC; ++w)
                acc_s[g][w][b] = y[g][w][b] = make_double2(0.0, 0.0);
        }

    auto columns = [&](auto plain) {
        for (int ig = threadIdx.x; ig < nc; ig += THREADS) {
            double2 a[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) a[b] = __ldg(nrow[b] + ig);
#pragma unroll
            for (int g = 0; g < RG; ++g) {
                const double2 wt = __ldg(wrow[g] + ig);
                const double2 ie = __ldg(erow[g] + ig);
                double2 A[NB], Aw[NB], B[NB];
                double wti2, awt2;
                flag_products<NB>(wt, ie, a, wti2, awt2, A, Aw, B);
                // Inf and NaN compare above the bound.
                const bool in_all = (unsigned long long)__double_as_longlong(awt2) <=
                                    (unsigned long long)__double_as_longlong(bound);
                if (any_most && in_all) {
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        all[g][b] = make_double2(__dadd_rn(all[g][b].x, B[b].x),
                                                 __dadd_rn(all[g][b].y, B[b].y));
                }
#pragma unroll
                for (int w = 0; w < NWC; ++w)
                    flag_term<NB, decltype(plain)::value>(f[w], in_all, wt, wti2, awt2, A, Aw, B, acc_s[g][w], y[g][w]);
            }
        }
    };
    if (all_plain)
        columns(std::true_type());
    else
        columns(std::false_type());

    double v[K];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int g = 0; g < RG; ++g)
#pragma unroll
            for (int w = 0; w < NWC; ++w) {
                const int k = b * KB + (g * NWC + w) * 4;
                double2 t = y[g][w][b];
                if (f[w].most)
                    t = make_double2(__dadd_rn(t.x, all[g][b].x), __dadd_rn(t.y, all[g][b].y));
                v[k] = acc_s[g][w][b].x;
                v[k + 1] = acc_s[g][w][b].y;
                v[k + 2] = flag_ssx_scale(f[w], t.x);
                v[k + 3] = flag_ssx_scale(f[w], t.y);
            }
    block_reduce<K, THREADS>(v, red, S);
#pragma unroll
    for (int b = 0; b < NB; ++b)
        if (band0 + b < p.nv)
            flag_epilogue<RG, NWC>(p, part, S + b * KB, row0, band0 + b, iw0,
                                   (long long)(band0 + b) * row_tiles + row_tile, row_tile);
}

}  // namespace gpp
