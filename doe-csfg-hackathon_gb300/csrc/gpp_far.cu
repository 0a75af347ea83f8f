// gpp_far.cu -- unoccupied bands with per-band frequencies: the terms whose
// frequency lies away from wtilde through a series, as products on the tensor
// cores.
//
// An unoccupied term is c aqsn Q / (wx - wtilde).  The plasmon-pole
// frequencies wtilde of a state lie in a band (a box of the complex plane,
// centre z0, half width h after a margin), while wx = E - E_n1 runs over the
// whole spectrum, so for most (band, frequency) pairs wx is well outside the
// box, and there, with u = (wx - z0) / h, z = (wtilde - z0) / h and
// r = u + sign(u) sqrt(u^2 - 1),
//
//   1 / (u - z) = (1 + 2 sum_{k >= 1} T_k(z) r^-k) / (r - u)
//
// (the generating function of the Chebyshev polynomials).  The sum over
// columns of a pair is then
//
//   sum_ig aqsn Q / (wx - wtilde) = sum_k b_k(wx) H_k,  H_k[n1][r] = sum_ig aqsn[n1][ig] P_k[r][ig],
//
// P_k = Q T_k(z): one complex product per k that every frequency of a band
// shares, instead of a division per (band, row, column, frequency).  |T_k| is
// at most rho^k on the box (rho: its Bernstein ellipse); a pair is `far` when
// |r| >= R rho, so the terms fall off by R and K = bits / log2 R of them reach
// the working precision; a band whose wx all lie further off needs fewer, and
// the bands are put in the order of what they need, so that the products of a
// term stop at the bands that have it.  The products run as residues
// (gpp_crt.cu), each k at the level of precision that R^-k leaves of the
// total's.
//
// What the series does not cover is computed term by term:
//  * near pairs (|r| < R rho, or a wx that is not finite): over every column,
//    in the call's precision;
//  * bands whose terms a fixed point does not hold (below): as near pairs;
//  * the columns whose wtilde lies outside the box (a few strays, such as
//    wtilde next to another band's frequency), for the far pairs, in FP64.
//
// The products' operands are fixed point, 57 bits of a row's largest value in
// each chunk of 512 columns, so their rounding is relative to max|aqsn| sum|Q| +
// sum|aqsn| max|Q| of a chunk, where term by term it is relative to the sum of
// |aqsn Q|.  The two differ where one factor is large just where the other is
// small.  So both are summed for every band first (weighted as the rows are;
// |aqsn| and |Q| in bf16, one product on the tensor cores), and a band whose
// ratio of the two passes kSpread is computed term by term: up to there the
// fixed point's rounding, about ratio 2^-57 of a term (all of the series' terms
// together), is no more than a term's in the per-term sums with their
// accumulation over the columns (2^-51).  Measured without the limit, 62 x 17 x
// 5003, FP64, at ratios of 3 to 87: 2.4e-16 of the band totals at all of them,
// per term 2.9e-16.  Uniform data gives 3 to 5, a chunk over which both factors
// fall by e^2 12.
//
// The box is chosen on the device from a histogram of Re(wtilde) against the
// histogram of wx, by the cost of what it leaves over; where no box pays, or
// too many columns or pairs are left over, the plan is inactive, every kernel
// here returns at once and the per-term kernel runs instead.  No host
// synchronisation; nothing depends on the order in which blocks run.
//
// GB300, FP64, 512 bands x 409 x 8192 x 3: 102.9 ms per term, 23-25 now (near
// pairs 15, products 3.2, terms 3.0, combine 1.6); mixed, 128 bands x 819 x 16384
// x 32: 120 ms per term, 36 now (near 23, terms 5.5, products 4.6); 512 bands x
// 1638 x 32768 x 3, 1% strays: 210 per term, 129 now (near 57, products 24,
// terms 19, strays 14, combine 13, spread 1.7).  The near kernels run at 1.25
// (FP64) and 1.4 (mixed) of the per-term kernels' time per pair: an entry holds
// 1.8 frequencies on average where a tile there shares its columns among 3.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "gpp_crt.h"
#include "gpp_crt_planes.cuh"
#include "gpp_far.h"
#include "gpp_tiles_fp64.cuh"

namespace gpp {

struct FarPlan {
    int active;
    int next;            // the near kernel's tile counter
    int planned;         // blocks of the plan that are done
    unsigned long long best;  // the best box so far: its cost's bits, and bins
    int n_near;
    long long n_out;
    int lo, hi;          // the box's bins of Re(wtilde)
    double x0, inv_w;    // bin = floor((x - x0) inv_w)
    double im_max;       // |Im(wtilde)| of a column in the box is at most this
    double z0, inv_h, h;
    double dfar;         // |wx - z0| of a far pair is at least this
    double log2_rho;
    int bands_at[64];    // bands whose series has a term k
    unsigned long long count[512];
    unsigned im[512];    // bits of the largest |Im| (float, rounded up) in each bin
};

namespace {

constexpr int kBins = 512;
constexpr int kNearTile = 4;  // entries per block of the FP64 near kernel
constexpr double kSpread = 64.0;

struct Sizes {
    int bands, ng, nc, nw;
    bool mixed;
    double R;
    double bits;         // what the series is cut at
    int K;               // its terms for a pair that is just far (at most 64)
    int Mp, ngp, nch, Kc;
    int gr;              // rows per group (a multiple of 8)
    int gm, slab;        // series terms and chunks per pass
    bool x_all;          // X's planes of every chunk at once
    int cap_near, near_rows;  // entries, row pairs per pass of the near kernel
    long long cap_out, seg_len;
    int segs;
    long long pairs;
    double c0;           // cost of the series at full occupancy, in per-term pairs
    float c0_call;       // as the call's sizes leave it (planes, launches, grids that do not fill)
    float near_least;    // near pairs that fill the near kernel's first round
};

// The scratch a call may take, apart from what has the size of an input or
// less: the planes and residues of a pass (with H, the sums they give, at most
// half as much again), the recurrence's state of a group of rows and X's planes
// half each, the near partials a quarter, the strays' an eighth.  A larger
// call runs in more passes.  GPP_SERIES_PASS_MB overrides it, for tests.
constexpr size_t kPassBytes = size_t(8) << 30;
size_t pass_bytes() {
    const char *v = getenv("GPP_SERIES_PASS_MB");
    const long long mb = v ? atoll(v) : 0;
    return mb > 0 ? (size_t)mb << 20 : kPassBytes;
}
size_t x_planes(int Mp, int Kc) { return (size_t)6 * kCrtN * Mp * Kc; }  // a chunk's

// Term k counts R^-k; three bits more past the first, so that all of them
// together round no worse than it does.
int level_of(const Sizes &z, int k) {
    const double need = (z.mixed ? 49.0 : 57.0) + (k > 0 ? 3.0 : 0.0) - k * std::log2(z.R);
    if (need > kCrtLevel[0].bits) return kCrtWide;
    int l = 0;
    while (l + 1 < kCrtWide && kCrtLevel[l + 1].bits >= need) ++l;
    return l;
}

Sizes sizes(const Problem &p, int bands, bool mixed) {
    Sizes z;
    z.bands = bands;
    z.ng = p.ng;
    z.nc = p.nc;
    z.nw = p.nw;
    z.mixed = mixed;
    z.bits = mixed ? 50.0 : 55.0;
    z.Mp = ceil_div(bands, kCrtRowsX) * kCrtRowsX;
    z.pairs = (long long)bands * p.nw;
    // Per cell: a per-term pair takes 20 ps (FP64) or 2.6 ps (mixed); a term of
    // the series 14 ps for its planes and 0.05 ps per padded band.
    const double term = (14.0 + 0.05 * z.Mp) / (mixed ? 2.6 : 20.0);
    // R balances the series' terms against the near pairs: where the terms are
    // a small part of the call a low R leaves fewer pairs near.  GB300: FP64
    // 512 x 409 x 8192 x 3, R = 2 / 2.25 / 2.5: 24.6 / 24.5 / 25.4 ms; mixed,
    // R = 2.5 / 3 / 4: 163 / 155 / 152 ms for 512 x 1638 x 32768 x 3 and
    // 64.6 / 64.3 / 68.0 ms for 128 x 819 x 16384 x 32.
    z.R = !mixed ? 2.25 : 32 * term > 0.25 * z.pairs ? 4.0 : 3.0;
    z.K = (int)std::ceil(z.bits / std::log2(z.R));
    z.c0 = z.K * term;
    z.ngp = ceil_div(p.ng, 8) * 8;
    z.near_least = mixed ? 0.f : 152.f * 4 * 1.8f / ceil_div(p.ng, 2);
    z.nch = std::max(1, ceil_div(p.nc, kCrtChunk));
    z.Kc = ceil_div(ceil_div(p.nc, z.nch), kCrtBlockK) * kCrtBlockK;
    // The same in time (ps), from the kernels' own rates: terms 14 a term and cell
    // from about 400 blocks on, the combination 0.018 a term, cell and band from
    // 760, the products 0.0316 a term, cell and padded band or the bytes of their
    // planes at 6 TB/s, X's planes 17 a level, band and column, the spread 30 a
    // value, and 150 us of launches.  FP64, 192 x 33 x 25601 x 1: 3.9 ms of these
    // and 1.8 of near pairs, which c0 put at 1.1 and 0.6 (per term 5.3); 420 x 17 x
    // 7937 x 3: 2.3 + 1.1 where per term takes 4.0.
    {
        const double cells = (double)z.ngp * p.nc, kt = z.K * cells, x = (double)z.Mp * p.nc;
        const double blocks = z.ngp / 8.0 * z.nch, quads = z.K / 5.0 * bands * z.ngp / 512;
        const double t = 14 * kt * std::max(1.0, 400 / blocks) + 0.018 * bands * kt * std::max(1.0, 760 / quads) +
                         std::max(0.0316 * z.Mp * kt, (64 * kt + 5 * 64 * x) / 6) + 5 * 17 * x +
                         30 * (cells + x) + 1.5e8;
        z.c0_call = (float)(t / ((mixed ? 2.6 : 20) * (double)p.ng * p.nc));
    }
    const size_t budget = pass_bytes();
    const size_t row_state = (size_t)(mixed ? 48 : 32) * z.nch * z.Kc;
    // Rows a group holds: their state, and four terms' planes and sums of a chunk.
    const size_t plane_rows = budget / (12 * (size_t)kCrtN * (2 * z.Kc + z.Mp)), sum_rows = budget / 2 / (64 * (size_t)bands);
    const size_t most = std::min({budget / 2 / row_state, plane_rows, sum_rows, (size_t)z.ngp});
    const int groups = ceil_div(z.ngp, (long long)std::max<size_t>(8, most / 8 * 8));
    z.gr = ceil_div(ceil_div(z.ngp, groups), 8) * 8;
    const size_t per = (size_t)3 * kCrtN * z.gr * (2 * (size_t)z.Kc + z.Mp);  // a term's, per chunk
    z.gm = (int)std::min<size_t>(z.K, std::max<size_t>(4, budget / (per * z.nch)));
    z.gm = (int)std::min<size_t>(z.gm, std::max<size_t>(1, budget / 2 / (16 * (size_t)bands * z.gr)));
    z.slab = (int)std::min<size_t>(z.nch, std::max<size_t>(1, budget / (per * z.gm)));
    z.x_all = x_planes(z.Mp, z.Kc) * z.nch <= budget / 2;
    if (!z.x_all) z.slab = (int)std::min<size_t>(z.slab, std::max<size_t>(1, budget / 2 / x_planes(z.Mp, z.Kc)));
    z.cap_near = (int)std::min<long long>(z.pairs / 2 + 1, 1 << 26);
    z.near_rows = (int)std::min<size_t>((p.ng + 1) / 2, std::max<size_t>(1, budget / 4 / (sizeof(double2) * kNearFreq * z.cap_near)));
    z.cap_out = (long long)p.ng * p.nc / 32 + 1;
    const long long segs = std::max<long long>(1, std::min<long long>(512, (long long)(budget / 8 / (sizeof(double2) * z.pairs))));
    z.seg_len = std::max<long long>(2048, (z.cap_out + segs - 1) / segs);
    z.segs = (int)((z.cap_out + z.seg_len - 1) / z.seg_len);
    return z;
}

struct Buffers {
    FarPlan *plan;
    int4 *near;
    int *place;        // [kNearFreq bands + 1]: a band's first entry of each length
    int *rows;         // [ng + 1]: strays before each row
    int2 *out;         // (row, column)
    double2 *C;        // [bands][ng]
    double2 *S1;       // [bands][K]
    double2 *near_part, *near_val, *out_part;
    void *state;       // P_(k-1), P_k (mixed: and z) between passes
    int *E0, *EA, *EX, *EY;
    float *SQ, *SA;      // [chunks][rows], [chunks][Mp]: sums of |Q|, |aqsn| over the chunk's exponent
    double2 *spread;     // per band: what the fixed point's rounding is relative to, and the sum of |aqsn Q|
    int *terms, *order;  // per band: its terms; the bands by their terms
    __nv_bfloat16 *sx, *sy;
    unsigned char *res;
    double2 *H;        // [bands][gm rows of a group]
};

size_t carve(const Sizes &z, void *ws, Buffers *b) {
    char *w = static_cast<char *>(ws);
    size_t off = 0;
    auto take = [&](size_t n) {
        char *q = w + off;
        off = align_up(off + n);
        return q;
    };
    Buffers o;
    const int Np = ceil_div((long long)z.gm * z.gr, kCrtRowsY) * kCrtRowsY;
    o.plan = reinterpret_cast<FarPlan *>(take(sizeof(FarPlan)));
    o.near = reinterpret_cast<int4 *>(take(sizeof(int4) * (size_t)z.cap_near));
    o.place = reinterpret_cast<int *>(take(sizeof(int) * ((size_t)kNearFreq * z.bands + 1)));
    o.rows = reinterpret_cast<int *>(take(sizeof(int) * ((size_t)z.ng + 1)));
    o.out = reinterpret_cast<int2 *>(take(sizeof(int2) * (size_t)z.cap_out));
    o.C = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)z.bands * z.ng));
    o.S1 = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)z.bands * z.K));
    o.near_part = reinterpret_cast<double2 *>(take(sizeof(double2) * kNearFreq * (size_t)z.cap_near * z.near_rows));
    o.near_val = reinterpret_cast<double2 *>(take(sizeof(double2) * kNearFreq * (size_t)z.cap_near));
    o.out_part = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)z.segs * z.pairs));
    o.state = take(sizeof(double2) * (z.mixed ? 3 : 2) * (size_t)z.nch * z.gr * z.Kc);
    o.terms = reinterpret_cast<int *>(take(sizeof(int) * (size_t)z.bands));
    o.order = reinterpret_cast<int *>(take(sizeof(int) * (size_t)z.bands));
    o.E0 = reinterpret_cast<int *>(take(sizeof(int) * (size_t)z.nch * z.ngp));
    o.EA = reinterpret_cast<int *>(take(sizeof(int) * (size_t)z.nch * z.Mp));
    o.SQ = reinterpret_cast<float *>(take(sizeof(float) * (size_t)z.nch * z.ngp));
    o.SA = reinterpret_cast<float *>(take(sizeof(float) * (size_t)z.nch * z.Mp));
    o.spread = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)z.bands));
    o.EX = reinterpret_cast<int *>(take(sizeof(int) * (size_t)z.nch * z.Mp));
    o.EY = reinterpret_cast<int *>(take(sizeof(int) * (size_t)z.slab * Np));
    o.sx = reinterpret_cast<__nv_bfloat16 *>(
        take(x_planes(z.Mp, z.Kc) * (z.x_all ? z.nch : z.slab)));
    o.sy = reinterpret_cast<__nv_bfloat16 *>(
        take(sizeof(__nv_bfloat16) * 3 * kCrtN * (size_t)Np * z.slab * z.Kc));
    o.res = reinterpret_cast<unsigned char *>(take((size_t)z.slab * 3 * kCrtN * z.Mp * Np));
    o.H = reinterpret_cast<double2 *>(take(sizeof(double2) * (size_t)z.bands * z.gm * z.gr));
    if (b) *b = o;
    return off;
}

__device__ __forceinline__ bool is_finite(double x) {
    return (__double2hiint(x) & 0x7FF00000) != 0x7FF00000;
}
// The bin of Re(wtilde), or -1 for a value outside the bins, an imaginary
// part above the cap or one that is not finite.
__device__ __forceinline__ int bin_of(const FarPlan &f, double2 wt) {
    if (!is_finite(wt.x) || !(fabs(wt.y) <= f.im_max)) return -1;
    const double t = (wt.x - f.x0) * f.inv_w;
    return t >= 0.0 && t < (double)kBins ? (int)t : -1;
}
__device__ __forceinline__ bool in_box(const FarPlan &f, double2 wt) {
    const int b = bin_of(f, wt);
    return b >= f.lo && b <= f.hi;
}
// Whether a band (its `spread`) is summed by the series at all, and a
// frequency of such a band.
__device__ __forceinline__ bool held(double2 spread) { return spread.x <= kSpread * spread.y; }
__device__ __forceinline__ bool is_far(const FarPlan &f, double wx) {
    return is_finite(wx) && fabs(wx - f.z0) >= f.dfar;
}

// The bins: 512 over the range of the unoccupied bands' finite wx with a
// margin, |Im(wtilde)| capped at 1/32 of it.
__global__ void __launch_bounds__(1024) far_range_kernel(Problem p, int b0, int bands, FarPlan *f) {
    __shared__ double lo[32], hi[32];
    double a = 1.0 / 0.0, b = -1.0 / 0.0;
    const unsigned n = (unsigned)bands * p.nw;  // below 2^20
    for (unsigned i = threadIdx.x; i < n; i += 1024) {
        const double x = p.wx[(size_t)(b0 + i / p.nw) * p.wx_stride + i % p.nw];
        if (is_finite(x)) {
            a = fmin(a, x);
            b = fmax(b, x);
        }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        a = fmin(a, __shfl_xor_sync(0xffffffffu, a, s));
        b = fmax(b, __shfl_xor_sync(0xffffffffu, b, s));
    }
    if ((threadIdx.x & 31) == 0) {
        lo[threadIdx.x >> 5] = a;
        hi[threadIdx.x >> 5] = b;
    }
    for (int i = threadIdx.x; i < kBins; i += 1024) {
        f->count[i] = 0;
        f->im[i] = 0;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    a = lo[threadIdx.x];
    b = hi[threadIdx.x];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        a = fmin(a, __shfl_xor_sync(0xffffffffu, a, s));
        b = fmax(b, __shfl_xor_sync(0xffffffffu, b, s));
    }
    if (threadIdx.x == 0) {
        f->active = f->n_near = f->next = f->planned = 0;
        f->n_out = 0;
        f->best = ~0ull;
        const double margin = 0.02 * (b - a) + 1e-3 * fmax(fabs(a), fabs(b));
        const double width = b - a + 2.0 * margin;
        // No finite wx, all zero, or a range past what the bins can divide: no bins.
        const bool ok = a <= b && width > 1e-100 && width < 1e100;
        f->x0 = ok ? a - margin : 0.0;
        f->inv_w = ok ? kBins / width : 0.0;
        f->im_max = ok ? width / 32.0 : -1.0;
    }
}

__global__ void __launch_bounds__(256) far_hist_kernel(Problem p, FarPlan *f) {
    __shared__ unsigned cnt[kBins], im[kBins];
    for (int i = threadIdx.x; i < kBins; i += 256) cnt[i] = im[i] = 0;
    const double x0 = f->x0, inv_w = f->inv_w, cap = f->im_max;
    __syncthreads();
    const size_t n = (size_t)p.ng * p.nc;
    FarPlan g;
    g.x0 = x0;
    g.inv_w = inv_w;
    g.im_max = cap;
#pragma unroll 4
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
        const double2 wt = __ldg(p.wt + i);
        const int b = bin_of(g, wt);
        if (b >= 0) {
            atomicAdd(&cnt[b], 1u);
            const unsigned v = __float_as_uint(__double2float_ru(fabs(wt.y)));
            if (v > im[b]) atomicMax(&im[b], v);  // a stale read only repeats the atomic
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBins; i += 256) {
        if (cnt[i]) atomicAdd(&f->count[i], (unsigned long long)cnt[i]);
        if (im[i]) atomicMax(&f->im[i], im[i]);
    }
}

// The box a .. b (bins lo .. hi, largest |Im| v): its half width after a
// margin, and the log2 of its ellipse.
struct Box {
    float z0, h, rho;
};
__device__ __forceinline__ Box box_of(float a, float b, float v) {
    Box q;
    const float hw = 0.5f * (b - a);
    q.z0 = 0.5f * (a + b);
    q.h = fmaxf(hw + v, 1.02f * hw);
    const float x = hw / q.h, y = v / q.h;
    // Sum of the distances from the corner to the foci: the largest on the box.
    const float s = 0.5f * (sqrtf((x - 1.f) * (x - 1.f) + y * y) + sqrtf((x + 1.f) * (x + 1.f) + y * y));
    q.rho = s + sqrtf(fmaxf(s * s - 1.f, 0.f));
    return q;
}

// Chooses the box.  The cost of a box is what it leaves to the per-term
// kernels, in pairs over all columns: its near pairs (times w_near), and the
// strays' share of the far ones (times w_out).  A warp takes one first bin, its
// lanes the last bins; the block that ends last takes the cheapest box of all
// (the smallest key, whatever the order).  Where no box pays, this and the
// launches that then return at once are what the series costs the call: with
// one block for the choice, 64 us of 4.3 ms.
constexpr int kPlanBlocks = kBins / 16;
__global__ void __launch_bounds__(kBins) far_plan_kernel(Problem p, int b0, int bands, FarPlan *f,
                                                         long long cap_out, float R, float c0,
                                                         float w_near, float near_least, float w_out) {
    __shared__ unsigned long long pre[kBins + 1], warp_cells[kBins / 32];
    __shared__ unsigned pairs_in[kBins], ppre[kBins + 1], warp_pairs[kBins / 32];
    __shared__ float vb[kBins];
    __shared__ int outside, last;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned n = (unsigned)bands * p.nw;
    const long long cells = (long long)p.ng * p.nc;
    if (t == 0) outside = 0;
    pairs_in[t] = 0;
    vb[t] = __uint_as_float(f->im[t]);
    __syncthreads();
    for (unsigned i = t; i < n; i += kBins) {
        const double x = p.wx[(size_t)(b0 + i / p.nw) * p.wx_stride + i % p.nw];
        const int b = bin_of(*f, make_double2(x, 0.0));
        if (b >= 0)
            atomicAdd(&pairs_in[b], 1u);
        else
            atomicAdd(&outside, 1);  // not finite: always near
    }
    __syncthreads();
    // Cells and pairs before each bin.
    unsigned long long c = f->count[t];
    unsigned q = pairs_in[t];
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const unsigned long long uc = __shfl_up_sync(0xffffffffu, c, s);
        const unsigned uq = __shfl_up_sync(0xffffffffu, q, s);
        if (lane >= s) {
            c += uc;
            q += uq;
        }
    }
    if (lane == 31) {
        warp_cells[warp] = c;
        warp_pairs[warp] = q;
    }
    __syncthreads();
    for (int k = 0; k < warp; ++k) {
        c += warp_cells[k];
        q += warp_pairs[k];
    }
    pre[t + 1] = c;
    ppre[t + 1] = q;
    if (t == 0) pre[0] = ppre[0] = 0;
    __syncthreads();
    const float w = (float)(1.0 / f->inv_w), total = (float)n, ncells = (float)cells;
    const int lo = blockIdx.x * (kBins / 32) + warp;
    unsigned long long mine = ~0ull;
    if (pre[lo + 1] > pre[lo] && f->inv_w > 0.0) {
        float before = 0.f;  // the largest |Im| of the bins lo .. j0 - 1
        for (int j0 = lo; j0 < kBins; j0 += 32) {
            const int j = j0 + lane;
            float v = j < kBins ? vb[j] : 0.f;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const float u = __shfl_up_sync(0xffffffffu, v, s);
                if (lane >= s) v = fmaxf(v, u);
            }
            v = fmaxf(v, before);
            before = __shfl_sync(0xffffffffu, v, 31);
            if (j >= kBins || pre[j + 1] == pre[j]) continue;
            const long long out = cells - (long long)(pre[j + 1] - pre[lo]);
            if (out > cap_out) continue;
            const Box bx = box_of(lo * w, (j + 1) * w, v);
            const float r = R * bx.rho, d = bx.h * 0.5f * (r + 1.f / r);
            const int i0 = max(0, min(kBins, (int)floorf((bx.z0 - d) / w)));
            const int i1 = max(0, min(kBins, (int)floorf((bx.z0 + d) / w) + 1));
            const float nr = (float)(ppre[i1] - ppre[i0]) + (float)outside;
            const float cost = (nr > 0.f ? fmaxf(nr, near_least) : 0.f) * w_near + (float)out / ncells * (total - nr) * w_out;
            const unsigned long long key =
                ((unsigned long long)__float_as_uint(fmaxf(cost, 0.f)) << 32) | (unsigned)(lo * kBins + j);
            if (key < mine) mine = key;
        }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) mine = min(mine, __shfl_xor_sync(0xffffffffu, mine, s));
    if (lane == 0 && mine != ~0ull) atomicMin(&f->best, mine);
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(&f->planned, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last || warp != 0) return;
    __threadfence();
    mine = *static_cast<volatile unsigned long long *>(&f->best);
    if (mine == ~0ull || !(__uint_as_float((unsigned)(mine >> 32)) + c0 < 0.9f * total)) return;
    const int a0 = (int)((unsigned)mine / kBins), a1 = (int)((unsigned)mine % kBins);
    float v = 0.f;
    for (int j = a0 + lane; j <= a1; j += 32) v = fmaxf(v, vb[j]);
    v = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
    if (lane != 0) return;
    const Box bx = box_of(a0 * w, (a1 + 1) * w, v);
    f->lo = a0;
    f->hi = a1;
    f->n_out = cells - (long long)(pre[a1 + 1] - pre[a0]);
    // In double, with margins above the float rounding of the choice.
    const double a = f->x0 + a0 / f->inv_w, b = f->x0 + (a1 + 1) / f->inv_w;
    f->z0 = 0.5 * (a + b);
    f->h = fmax((double)bx.h, 0.5 * (b - a));
    f->inv_h = 1.0 / f->h;
    const double rho = (double)bx.rho * 1.00001, r = (double)R * rho;
    f->log2_rho = log2(rho);
    f->dfar = f->h * 0.5 * (r + 1.0 / r);
    f->active = 1;
}

// An entry of the near list covers up to kNearFreq consecutive near
// frequencies of a band: every kNearFreq-th pair of a run of them starts one.
// A warp walks band n's frequencies and calls found(start, iw, len) for each 32
// of them, all lanes together: whether lane's frequency iw starts an entry, and
// of which length.
template <class Found>
__device__ __forceinline__ void near_runs(const Problem &p, const FarPlan &f, int band, bool far_band,
                                          Found found) {
    const int lane = threadIdx.x & 31;
    const double *wx = p.wx + (size_t)band * p.wx_stride;
    int carry = 0;  // the run that reaches the first of these 32
    for (int w0 = 0; w0 < p.nw; w0 += 32) {
        const int iw = w0 + lane;
        const unsigned m = __ballot_sync(0xffffffffu, iw < p.nw && !(far_band && is_far(f, wx[min(iw, p.nw - 1)])));
        const unsigned gaps = ~m & ((1u << lane) - 1);
        const int before = gaps ? lane - 32 + __clz(gaps) : lane + carry;
        const bool start = ((m >> lane) & 1) && before % kNearFreq == 0;
        int len = 1;
        if (start)
            while (len < kNearFreq && iw + len < p.nw && !(far_band && is_far(f, wx[iw + len]))) ++len;
        found(start, iw, len);
        carry = m == 0xffffffffu ? carry + 32 : __clz(~m);
    }
}
// Entries of each length per band: count[l bands + n], l = kNearFreq - length.
__global__ void __launch_bounds__(256) far_near_count_kernel(Problem p, const FarPlan *f, int b0,
                                                             int bands, const double2 *spread, int *count) {
    if (!f->active) return;
    const int n = (blockIdx.x * 256 + threadIdx.x) >> 5;
    if (n >= bands) return;
    int c[kNearFreq] = {};
    near_runs(p, *f, b0 + n, held(spread[n]), [&](bool start, int, int len) {
#pragma unroll
        for (int l = 0; l < kNearFreq; ++l)
            c[l] += __popc(__ballot_sync(0xffffffffu, start && len == kNearFreq - l));
    });
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int l = 0; l < kNearFreq; ++l) count[l * bands + n] = c[l];
}
// The counts become places, the longest entries first, so that the warps of a
// block have equal work; the plan is dropped if too many pairs are near.
__global__ void __launch_bounds__(1024) far_near_scan_kernel(FarPlan *f, int bands, int nw, int *count,
                                                             int cap_near, float c0, float w_near,
                                                             float near_least) {
    if (!f->active) return;
    __shared__ int part[1024];
    __shared__ unsigned long long pairs;
    const int n = kNearFreq * bands, per = (n + 1023) / 1024;
    const int a = threadIdx.x * per, b = min(n, a + per);
    if (threadIdx.x == 0) pairs = 0;
    __syncthreads();
    int s = 0;
    unsigned long long q = 0;
    for (int i = a; i < b; ++i) {
        s += count[i];
        q += (unsigned long long)count[i] * (kNearFreq - i / bands);
    }
    part[threadIdx.x] = s;
    if (q) atomicAdd(&pairs, q);
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int i = 0; i < 1024; ++i) {
            const int v = part[i];
            part[i] = acc;
            acc += v;
        }
        const float total = (float)((long long)bands * nw);
        if (pairs > (unsigned long long)cap_near || fmaxf((float)pairs, near_least) * w_near + c0 >= 0.95f * total)
            f->active = 0;
        f->n_near = acc;
        count[n] = acc;
    }
    __syncthreads();
    s = part[threadIdx.x];
    for (int i = a; i < b; ++i) {
        const int v = count[i];
        count[i] = s;
        s += v;
    }
}
__global__ void __launch_bounds__(256) far_near_list_kernel(Problem p, const FarPlan *f, int b0,
                                                            int bands, const double2 *spread,
                                                            const int *place, int4 *near) {
    if (!f->active) return;
    const int n = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (n >= bands) return;
    int at[kNearFreq];
#pragma unroll
    for (int l = 0; l < kNearFreq; ++l) at[l] = place[l * bands + n];
    near_runs(p, *f, b0 + n, held(spread[n]), [&](bool start, int iw, int len) {
#pragma unroll
        for (int l = 0; l < kNearFreq; ++l) {
            const bool mine = start && len == kNearFreq - l;
            const unsigned m = __ballot_sync(0xffffffffu, mine);
            if (mine) near[at[l] + __popc(m & ((1u << lane) - 1))] = make_int4(b0 + n, iw, len, 0);
            at[l] += __popc(m);
        }
    });
}

// Terms each band's series needs (for the nearest of its far frequencies; 0
// without one), and the bands by that number, the most first, in band order
// where it is equal.  Past kOrderBands the bands keep their order and all
// terms.
constexpr int kOrderBands = 8192;
__global__ void __launch_bounds__(256) far_need_kernel(Problem p, FarPlan *f, int b0, int bands,
                                                       int K, double bits, const double2 *spread,
                                                       int *terms) {
    if (!f->active) return;
    if (blockIdx.x == 0 && threadIdx.x < 64)
        f->bands_at[threadIdx.x] = bands > kOrderBands && (int)threadIdx.x < K ? bands : 0;
    const int n = blockIdx.x * 256 + threadIdx.x;
    if (n >= bands) return;
    double d = 1.0 / 0.0;
    for (int w = 0; held(spread[n]) && w < p.nw; ++w) {
        const double x = p.wx[(size_t)(b0 + n) * p.wx_stride + w];
        if (is_far(*f, x)) d = fmin(d, fabs(x - f->z0));
    }
    int k = 0;
    if (d < 1e300) {
        const double u = d * f->inv_h, lr = log2(u + sqrt((u - 1.0) * (u + 1.0))) - f->log2_rho;
        k = min(K, (int)ceil(bits / lr));
    }
    terms[n] = bands > kOrderBands ? K : k;
}
__global__ void __launch_bounds__(256) far_order_kernel(FarPlan *f, int bands, const int *terms,
                                                        int *order) {
    if (!f->active) return;
    __shared__ int tile[256];
    const int n = blockIdx.x * 256 + threadIdx.x;
    if (bands > kOrderBands) {
        if (n < bands) order[n] = n;
        return;
    }
    const int mine = n < bands ? terms[n] : 0;
    int rank = 0;
    for (int t0 = 0; t0 < bands; t0 += 256) {
        tile[threadIdx.x] = t0 + (int)threadIdx.x < bands ? terms[t0 + threadIdx.x] : -1;
        __syncthreads();
        for (int i = 0; i < 256; ++i) rank += tile[i] > mine || (tile[i] == mine && t0 + i < n);
        __syncthreads();
    }
    if (n < bands) order[rank] = n;
    // Bands with a term k: those with more than k terms.
    if (n < bands)
        for (int k = 0; k < mine; ++k) atomicAdd(&f->bands_at[k], 1);
}

// Strays per row, their offsets, and their (row, column) list in order.
__global__ void __launch_bounds__(256) far_count_kernel(Problem p, const FarPlan *f, int *rows) {
    if (!f->active || f->n_out == 0) return;
    __shared__ int c[8];
    const int r = blockIdx.x;
    int n = 0;
    for (int ig = threadIdx.x; ig < p.nc; ig += 256) n += !in_box(*f, __ldg(p.wt + (size_t)r * p.nc + ig));
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0) c[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) n += c[w];
        rows[r + 1] = n;
    }
}
__global__ void __launch_bounds__(1024) far_scan_kernel(int ng, const FarPlan *f, int *rows) {
    if (!f->active || f->n_out == 0) return;
    __shared__ int part[1024];
    const int per = (ng + 1023) / 1024, a = threadIdx.x * per, b = min(ng, a + per);
    int s = 0;
    for (int i = a; i < b; ++i) s += rows[i + 1];
    part[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int i = 0; i < 1024; ++i) {
            const int v = part[i];
            part[i] = acc;
            acc += v;
        }
        rows[0] = 0;
    }
    __syncthreads();
    s = part[threadIdx.x];
    for (int i = a; i < b; ++i) rows[i + 1] = s += rows[i + 1];
}
__global__ void __launch_bounds__(256) far_list_kernel(Problem p, const FarPlan *f, const int *rows,
                                                       int2 *out) {
    if (!f->active || f->n_out == 0) return;
    __shared__ int c[8];
    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int at = rows[r];
    if (rows[r + 1] == at) return;
    for (int g0 = 0; g0 < p.nc; g0 += 256) {
        const int ig = g0 + threadIdx.x;
        const bool is = ig < p.nc && !in_box(*f, __ldg(p.wt + (size_t)r * p.nc + ig));
        const unsigned m = __ballot_sync(0xffffffffu, is);
        if (lane == 0) c[warp] = __popc(m);
        __syncthreads();
        int k = at + __popc(m & ((1u << lane) - 1));
        int all = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            if (w < warp) k += c[w];
            all += c[w];
        }
        if (is) out[k] = make_int2(r, ig);
        at += all;
        __syncthreads();
    }
}

// c[k][r] = 0.5 vcoul conj(aqsm[b0 + k]) at row r's G' index (0 where that is
// invalid; the fault is recorded).
__global__ void __launch_bounds__(256) far_coeff_kernel(Problem p, int b0, int bands, double2 *C,
                                                        const FarPlan *f, int *err) {
    if (!f->active) return;
    const long long n = (long long)bands * p.ng;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const int k = (int)(i / p.ng), r = (int)(i % p.ng);
        const int igp = resolve_igp(p, r, err);
        double2 c = make_double2(0.0, 0.0);
        if (igp >= 0) {
            const double2 m = __ldg(p.aqsm + (size_t)(b0 + k) * p.nc + igp);
            c = cscale(make_double2(0.5 * m.x, -0.5 * m.y), __ldg(p.vcoul + igp));
        }
        C[i] = c;
    }
}

// round(x 2^(bits - e)) for bits <= 30 on 32-bit words, e >= 0, |x| < 2^e (a
// subnormal, then far below half a unit, counts as zero).
__device__ __forceinline__ int fixed_point32(double x, int e, int bits) {
    const unsigned hi = __double2hiint(x), lo = __double2loint(x);
    const int E = (hi >> 20) & 0x7FF;
    const unsigned mh = (hi & 0xFFFFFu) | 0x100000u;  // 53-bit mantissa, x = m 2^(E - 1075)
    // One bit more than the result, then rounded (ties away from zero).
    const int sh = 1074 - E - bits + e;
    unsigned n = 0;
    if (sh < 32)
        n = __funnelshift_r(lo, mh, sh);
    else if (sh < 64)
        n = mh >> (sh - 32);
    if (E == 0) n = 0;
    n = (n + 1) >> 1;
    return (int)hi < 0 ? -(int)n : (int)n;
}

// What the spread of a band is formed from: for 8 rows x one chunk the exponent
// E of the largest |re|, |im|, the magnitudes over 2^E in bf16 (core-matrix
// blocks of R rows) and their sum S.  Y: rows of Q, 0 outside the box; else
// rows of aqsn, from row b0 on; E and S have a row of ld per chunk.  A thread
// per 8 consecutive columns of a row, which it reads twice (from L2 the second
// time): Q in FP64 for its exponent and the box, then the magnitudes in float,
// |Q| as |wtilde| |I_eps| (1638 x 32768: 1.3 ms, bound by the first; 2.2 with
// both in FP64).
template <bool Y>
__global__ void __launch_bounds__(128) far_sizes_kernel(Problem p, const FarPlan *f, int b0, int L, int Lp,
                                                        int ld, int c0, int nc, int Kc, int *E, float *S,
                                                        __nv_bfloat16 *out) {
    constexpr int R = Y ? kCrtRowsY : kCrtRowsX;
    if (!f->active) return;
    __shared__ unsigned long long red[4][8];
    __shared__ float sum[4][8];
    __shared__ int exps[8];
    const int groups = Lp / 8, l0 = blockIdx.x % groups * 8, c = blockIdx.x / groups;
    const int t = threadIdx.x, row = t & 7, l = l0 + row, kb = (c0 + c) * Kc, end = min(p.nc, kb + Kc);
    const double2 *at = (Y ? p.wt : p.aqsn) + (size_t)(b0 + l) * p.nc, *ie = p.ieps + (size_t)(b0 + l) * p.nc;
    unsigned long long mx = 0;
    unsigned in = 0;  // the columns that count, in the order of the loops (at most 4 x 8)
    int bit = 0;
    for (int k = t >> 3; k < Kc / 8; k += 16)
#pragma unroll
        for (int j = 0; j < 8; ++j, ++bit) {
            const int ig = kb + k * 8 + j;
            if (l >= L || ig >= end) continue;
            double2 v = __ldg(at + ig);
            if constexpr (Y) {
                if (!in_box(*f, v)) continue;
                v = cmul(v, __ldg(ie + ig));
            }
            in |= 1u << bit;
            const unsigned long long a = (unsigned long long)__double_as_longlong(v.x) & 0x7FFFFFFFFFFFFFFFull;
            const unsigned long long b = (unsigned long long)__double_as_longlong(v.y) & 0x7FFFFFFFFFFFFFFFull;
            mx = max(mx, max(a, b));
        }
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
    if ((t & 24) == 0) red[t >> 5][row] = mx;
    __syncthreads();
    if (t < 8) {
        for (int w = 1; w < 4; ++w) mx = max(mx, red[w][t]);
        exps[t] = crt_exponent(mx);
        E[(size_t)(c0 + c) * ld + l0 + t] = exps[t];
    }
    __syncthreads();
    const int e = exps[row], ksteps = nc * (Kc / kCrtBlockK);
    __nv_bfloat16 *w0 = out + ((size_t)(l0 / R) * ksteps * (R / 8) + (size_t)(l0 % R) / 8) * 512 + row * 8;
    // |z| 2^-e2, each part from its bits (the top 20 of the mantissa), between
    // 2^-120 and 2^120.  wtilde is taken over the box's exponent eb, I_eps over
    // 2^(e - eb); near FP64's lower end by FP64.
    const int eb = Y ? ilogb(fabs(f->z0) + f->h) + 2 : 0;
    auto over = [&](double2 z, int e2) {
        float m[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double x = h ? z.y : z.x;
            const int hi = __double2hiint(x) & 0x7FFFFFFF, sh = min((hi >> 20) - 1022 - e2, 120);
            m[h] = e2 < -900 ? (float)fmin(fabs(ldexp(x, -e2)), 0x1p120)
                   : sh < -120 ? 0.f
                               : __int_as_float(((sh + 126) << 23) | ((hi & 0xFFFFF) << 3));
        }
        // Within 4% of the magnitude (a square would leave float's range).
        return fmaxf(0.96f * fmaxf(m[0], m[1]) + 0.4f * fminf(m[0], m[1]), fmaxf(m[0], m[1]));
    };
    if (e == kExpNonFinite || e == kExpZero) in = 0;
    bit = 0;
    float total = 0.f;
    for (int k = t >> 3; k < Kc / 8; k += 16) {
        unsigned v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float m[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                m[h] = 0.f;
                const int ig = kb + k * 8 + 2 * j + h;
                if ((in >> bit++) & 1) {
                    if constexpr (Y)
                        m[h] = over(__ldg(at + ig), eb) * over(__ldg(ie + ig), e - eb);
                    else
                        m[h] = over(__ldg(at + ig), e);
                }
            }
            const __nv_bfloat162 q = __floats2bfloat162_rn(m[0], m[1]);
            total += __low2float(q) + __high2float(q);
            v[j] = *reinterpret_cast<const unsigned *>(&q);
        }
        const int ks = c * (Kc / kCrtBlockK) + (k >> 3);
        *reinterpret_cast<uint4 *>(w0 + (size_t)ks * (R / 8) * 512 + (k & 7) * 64) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    total += __shfl_xor_sync(0xffffffffu, total, 8);
    total += __shfl_xor_sync(0xffffffffu, total, 16);
    if ((t & 24) == 0) sum[t >> 5][row] = total;
    __syncthreads();
    if (t < 8) S[(size_t)(c0 + c) * ld + l0 + t] = sum[0][t] + sum[1][t] + sum[2][t] + sum[3][t];
}

// spread[n] (+)= over the rows [r0, r0 + rows) and chunks [c0, c0 + nc): |c| 2^(EA + E0) times
// SA + SQ (the largest magnitudes count 1 each) and times V, the chunk's sum of
// products.  A row's chunks are summed in float over its largest E0 and the
// band's largest EA (512 x 1638 x 64 chunks: 0.26 ms, 1.0 in FP64).
__global__ void __launch_bounds__(256) far_spread_kernel(const FarPlan *f, const double2 *C, const int *EA,
                                                         const int *E0, const float *SA, const float *SQ,
                                                         const float *V, int ng, int ngp, int r0, int rows,
                                                         int Mp, int Np, int c0, int nc, int add,
                                                         double2 *spread) {
    if (!f->active) return;
    __shared__ double red[16], S[2];
    const int n = blockIdx.x;
    int ea = kExpZero;
    for (int c = 0; c < nc; ++c) ea = max(ea, EA[(size_t)(c0 + c) * Mp + n]);
    double v[2] = {0.0, 0.0};
    for (int r = threadIdx.x; r < rows; r += 256) {
        const int *e0 = E0 + (size_t)c0 * ngp + r0 + r;
        int er = kExpZero;
        for (int c = 0; c < nc; ++c) er = max(er, e0[(size_t)c * ngp]);
        float a = 0.f, b = 0.f;
        for (int c = 0; c < nc; ++c) {
            const size_t x = (size_t)(c0 + c) * Mp + n, y = (size_t)c * ngp;
            const int ex = EA[x] - ea + e0[y] - er;  // at most 0
            const float w = ex < -126 ? 0.f : __int_as_float((127 + ex) << 23);
            a = fmaf(w, SA[x] + SQ[(size_t)c0 * ngp + r0 + r + y], a);
            b = fmaf(w, V[((size_t)c * Mp + n) * Np + r], b);
        }
        const double2 z = C[(size_t)n * ng + r0 + r];
        const double m = scalbn(sqrt(z.x * z.x + z.y * z.y), ea + er);
        v[0] = fma(m, (double)a, v[0]);
        v[1] = fma(m, (double)b, v[1]);
    }
    block_reduce<2, 256>(v, red, S);
    if (threadIdx.x == 0) {
        const double2 old = add ? spread[n] : make_double2(0.0, 0.0);
        spread[n] = make_double2(old.x + S[0], old.y + S[1]);
    }
}

// Residue planes and exponents of P_k, k = k0 .. k0 + gm - 1, for 8 rows x one
// chunk at level L, of the gr rows from r0 on: row r0 + l of term m is row
// m gr + l of the product's Y operand, in the core-matrix blocks of
// crt_prep_kernel.  A thread carries 4 consecutive columns of a row (half a
// core-matrix row; 8 would halve the resident warps) through the recurrence
// P_(k+1) = 2 z P_k - P_(k-1) (P_-1 = z Q starts it) and leaves P_(k-1), P_k for
// the next pass in `state`.  The exponent of term k is that of the chunk's
// largest |re|, |im| of Q, raised by the bound rho^k of |T_k| and 1.  Q is scaled
// by the chunk's exponent first: the terms of a chunk at either end of FP64's
// range keep their precision.  Columns outside the box are zero.
//
// In mixed precision the recurrence runs in float-float (DF): FP64 kept its
// pipe 62-76% busy with 4 instructions per term and column where the residues
// take most of the issue slots.  1638 x 32768, 25 terms: 26 -> 19 ms.  Only the
// first pass reads the inputs, the next ones find z with the last two terms in
// `state`.
constexpr int kTermK = 4;  // columns per thread
template <int L, bool DF>
__global__ void __launch_bounds__(128, 4) far_terms_kernel(Problem p, const FarPlan *f, int ngp, int r0, int gr, int c0,
                                                           int nc, int Kc, int Np, int k0, int gm,
                                                           int last, __nv_bfloat16 *out, int *EY,
                                                           const int *E0, void *state) {
    constexpr int NMOD = kCrtLevel[L].n, BITS = kCrtLevel[L].bits, ND = BITS > 41 ? 4 : BITS > 18 ? 3 : 2;
    if (!f->active) return;
    __shared__ int exps[8];
    const int groups = gr / 8;
    const int grp = blockIdx.x % groups, c = blockIdx.x / groups;
    const int t = threadIdx.x, half = t & 1, row = (t >> 1) & 7, kg0 = t >> 4, l = grp * 8 + row, r = r0 + l;
    const int kb = (c0 + c) * Kc, items = (Kc + 63) / 64;
    const double2 *wrow = p.wt + (size_t)min(r, p.ng - 1) * p.nc;
    const double2 *erow = p.ieps + (size_t)min(r, p.ng - 1) * p.nc;
    const double z0 = f->z0, inv_h = f->inv_h;
    auto at = [&](int ig, double2 &wt) {
        if (r >= p.ng || ig >= p.nc) return false;
        wt = __ldg(wrow + ig);
        return in_box(*f, wt);
    };
    if (t < 8) exps[t] = E0[(size_t)(c0 + c) * ngp + r0 + grp * 8 + t];
    __syncthreads();
    const int e0 = exps[row];
    // x 2^-e0 in two exact steps (what is lost below 2^-1022 of the largest
    // value is far below the last bit).
    const int h0 = max(-2000, min(e0, 2000)) / 2, h1 = max(-2000, min(e0, 2000)) - h0;
    const double s0 = __hiloint2double((1023 - h0) << 20, 0), s1 = __hiloint2double((1023 - h1) << 20, 0);
    auto scaled = [&](double2 q) { return make_double2(q.x * s0 * s1, q.y * s0 * s1); };
    const double log2_rho = f->log2_rho;
    auto raise = [&](int k) { return k == 0 ? 0 : 1 + (int)ceil(k * log2_rho); };
    if (half == 0)
        for (int m = kg0; m < gm; m += 8) EY[(size_t)c * Np + (size_t)m * gr + l] = e0 + raise(k0 + m);

    const int ksteps = nc * (Kc / kCrtBlockK);
    const size_t plane = (size_t)Np * ksteps * kCrtBlockK;
    if constexpr (DF) {
        // Two pairs of columns per thread: z2, then P_(k-1) and P_k as df2.
        constexpr int NP = kTermK / 2;
        float4 *st = static_cast<float4 *>(state) + ((size_t)(c0 + c) * groups + grp) * (size_t)items * (NP * 6 * 128) + t;
        auto load = [&](size_t at) {
            const float4 v = st[at * 128];
            return df2{f2(v.x, v.y), f2(v.z, v.w)};
        };
        auto store = [&](size_t at, const df2 &v) {
            st[at * 128] = make_float4(v.h.x, v.h.y, v.l.x, v.l.y);
        };
        const bool finite = e0 != kExpZero && e0 != kExpNonFinite;
        for (int i = 0; i < items; ++i) {
            const int kg = kg0 + 8 * i;
            df2 zr[NP], zi[NP], cr[NP], ci[NP], pr[NP], pi[NP];
#pragma unroll
            for (int h = 0; h < NP; ++h) {
                const size_t at6 = (size_t)(i * NP + h) * 6;
                if (k0 > 0) {
                    zr[h] = load(at6), zi[h] = load(at6 + 1);
                    pr[h] = load(at6 + 2), pi[h] = load(at6 + 3);
                    cr[h] = load(at6 + 4), ci[h] = load(at6 + 5);
                    continue;
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int ig = kb + kg * 8 + half * kTermK + 2 * h + j;
                    double2 wt, z = make_double2(0.0, 0.0), q = z;
                    if (at(ig, wt) && finite) {
                        z = make_double2(2.0 * (wt.x - z0) * inv_h, 2.0 * wt.y * inv_h);
                        q = cmul(wt, __ldg(erow + ig));
                        q = scaled(q);
                    }
                    df2_set_lane(zr[h], j, split_bits(z.x));
                    df2_set_lane(zi[h], j, split_bits(z.y));
                    df2_set_lane(cr[h], j, split_bits(q.x));
                    df2_set_lane(ci[h], j, split_bits(q.y));
                }
                const df2 half_r = {f2mul(zr[h].h, f2(0.5f, 0.5f)), f2mul(zr[h].l, f2(0.5f, 0.5f))};
                const df2 half_i = {f2mul(zi[h].h, f2(0.5f, 0.5f)), f2mul(zi[h].l, f2(0.5f, 0.5f))};
                pr[h] = df2_norm(df2_sub(df2_mul(half_r, cr[h]), df2_mul(half_i, ci[h])));
                pi[h] = df2_norm(df2_add(df2_mul(half_r, ci[h]), df2_mul(half_i, cr[h])));
                if (!last) store(at6, zr[h]), store(at6 + 1, zi[h]);
            }
            const int ks = c * (Kc / kCrtBlockK) + i;
#pragma unroll 1
            for (int m = 0; m < gm; ++m) {
                const float scale = ldexpf(1.0f, BITS - raise(k0 + m));
                const int y = m * gr + grp * 8;
                __nv_bfloat16 *w = out + ((size_t)(y / kCrtRowsY) * ksteps + ks) * (kCrtRowsY * kCrtBlockK) +
                                   (size_t)((y % kCrtRowsY) / 8) * 512 + kg0 * 64 + row * 8 + half * kTermK;
                float2 dr[NP][ND], di[NP][ND];
#pragma unroll
                for (int h = 0; h < NP; ++h) {
                    crt_digits_df2<ND>(cr[h], scale, dr[h]);
                    crt_digits_df2<ND>(ci[h], scale, di[h]);
                }
                crt_store_residues<NP, ND>(dr, di, NMOD, w, plane);
#pragma unroll
                for (int h = 0; h < NP; ++h) {
                    const df2 nr = df2_norm(df2_sub(df2_mul(zr[h], cr[h]),
                                                    df2_add(df2_mul(zi[h], ci[h]), pr[h])));
                    const df2 ni = df2_norm(df2_add(df2_mul(zr[h], ci[h]),
                                                    df2_sub(df2_mul(zi[h], cr[h]), pi[h])));
                    pr[h] = cr[h], pi[h] = ci[h];
                    cr[h] = nr, ci[h] = ni;
                }
            }
            if (last) continue;
#pragma unroll
            for (int h = 0; h < NP; ++h) {
                const size_t at6 = (size_t)(i * NP + h) * 6;
                store(at6 + 2, pr[h]), store(at6 + 3, pi[h]);
                store(at6 + 4, cr[h]), store(at6 + 5, ci[h]);
            }
        }
        return;
    } else {
    double2 *st = static_cast<double2 *>(state) + ((size_t)(c0 + c) * groups + grp) * (size_t)items * (2 * kTermK * 128);
    for (int i = 0; i < items; ++i) {  // Kc is a multiple of 64: 8 k-cores per turn
        const int kg = kg0 + 8 * i;
        double2 cur[kTermK], prev[kTermK], z2[kTermK];
#pragma unroll
        for (int kk = 0; kk < kTermK; ++kk) {
            const int ig = kb + kg * 8 + half * kTermK + kk;
            double2 wt;
            const bool in = at(ig, wt);
            z2[kk] = in ? make_double2(2.0 * (wt.x - z0) * inv_h, 2.0 * wt.y * inv_h)
                        : make_double2(0.0, 0.0);
            if (k0 == 0) {
                cur[kk] = in ? scaled(cmul(wt, __ldg(erow + ig))) : make_double2(0.0, 0.0);
                const double2 d = cmul(cur[kk], z2[kk]);
                prev[kk] = make_double2(0.5 * d.x, 0.5 * d.y);
            } else {
                prev[kk] = st[((size_t)(i * kTermK + kk) * 2) * 128 + t];
                cur[kk] = st[((size_t)(i * kTermK + kk) * 2 + 1) * 128 + t];
            }
        }
        const int ks = c * (Kc / kCrtBlockK) + i;
#pragma unroll 1
        for (int m = 0; m < gm; ++m) {
            const int e = raise(k0 + m);
            const int y = m * gr + grp * 8;
            __nv_bfloat16 *w = out + ((size_t)(y / kCrtRowsY) * ksteps + ks) * (kCrtRowsY * kCrtBlockK) +
                               (size_t)((y % kCrtRowsY) / 8) * 512 + kg0 * 64 + row * 8 + half * kTermK;
            float2 dr[kTermK / 2][ND], di[kTermK / 2][ND];
            auto digits = [&](double x, float(&d)[ND]) {
                if constexpr (BITS <= 30)
                    crt_digits_n<ND>(fixed_point32(x, e, BITS), d);
                else
                    crt_digits_n<ND>(oz_fixed_point(x, e, BITS), d);
            };
#pragma unroll
            for (int h = 0; h < kTermK / 2; ++h) {
                float a[ND], b[ND], x[ND], v[ND];
                digits(cur[2 * h].x, a);
                digits(cur[2 * h + 1].x, b);
                digits(cur[2 * h].y, x);
                digits(cur[2 * h + 1].y, v);
#pragma unroll
                for (int k = 0; k < ND; ++k) {
                    dr[h][k] = f2(a[k], b[k]);
                    di[h][k] = f2(x[k], v[k]);
                }
            }
            crt_store_residues<kTermK / 2, ND>(dr, di, NMOD, w, plane);
#pragma unroll
            for (int kk = 0; kk < kTermK; ++kk) {
                const double2 n = make_double2(
                    fma(z2[kk].x, cur[kk].x, fma(-z2[kk].y, cur[kk].y, -prev[kk].x)),
                    fma(z2[kk].x, cur[kk].y, fma(z2[kk].y, cur[kk].x, -prev[kk].y)));
                prev[kk] = cur[kk];
                cur[kk] = n;
            }
        }
        if (!last) {
#pragma unroll
            for (int kk = 0; kk < kTermK; ++kk) {
                st[((size_t)(i * kTermK + kk) * 2) * 128 + t] = prev[kk];
                st[((size_t)(i * kTermK + kk) * 2 + 1) * 128 + t] = cur[kk];
            }
        }
    }
    }
}

// S1[n][k0 + m] (+)= sum over l < rows of c[n][r0 + l] H[.][m gr + l] for the
// band n at place blockIdx.x of the order; 0 for a band without the term.
__global__ void __launch_bounds__(256) far_fold_kernel(const FarPlan *f, const int *order,
                                                       const double2 *C, const double2 *H, int ng,
                                                       int r0, int rows, int gr, int ld, int k0, int K,
                                                       double2 *S1) {
    if (!f->active) return;
    __shared__ double red[16], S[2];
    const int at = blockIdx.x, n = order[at], m = blockIdx.y;
    double v[2] = {0.0, 0.0};
    if (at >= f->bands_at[k0 + m]) {
        if (threadIdx.x == 0) S1[(size_t)n * K + k0 + m] = make_double2(0.0, 0.0);
        return;
    }
    for (int l = threadIdx.x; l < rows; l += 256) {
        const double2 x = cmul(C[(size_t)n * ng + r0 + l], H[(size_t)at * ld + (size_t)m * gr + l]);
        v[0] += x.x;
        v[1] += x.y;
    }
    block_reduce<2, 256>(v, red, S);
    if (threadIdx.x == 0) {
        double2 *o = S1 + (size_t)n * K + k0 + m;
        *o = r0 ? cadd(*o, make_double2(S[0], S[1])) : make_double2(S[0], S[1]);
    }
}

// Near pairs in FP64: a block takes a row pair x kNearTile entries, threads
// striding over the columns as in noflag_fp64_tile; each entry's weighted sums
// of the two rows go to partial[entry][frequency][row pair].
__global__ void __launch_bounds__(128) far_near_fp64_kernel(Problem p, FarNear nr) {
    constexpr int RN = kNearTile, NF = kNearFreq, K = RN * 2 * NF * 2;
    __shared__ double red[4 * K], S[K];
    if (!*nr.active) return;
    const int count = *nr.count, tiles = (count + RN - 1) / RN, pairs = nr.pairs;
    const int nc = p.nc;
    constexpr int kRows = 16;  // row pairs in L2 while the entries stream past them
    __shared__ int item;
    for (;;) {  // tiles differ in length: blocks take them from a counter
        if (threadIdx.x == 0) item = atomicAdd(nr.next, 1);
        __syncthreads();
        const long long b = item;
        if (b >= (long long)tiles * pairs) break;
        const long long per = (long long)kRows * tiles;
        const int g = (int)(b / per), in = (int)(b % per);
        const int here = min(kRows, pairs - g * kRows);
        const int rp = nr.pair0 + g * kRows + in % here, e0 = in / here * RN;
        const double2 *wr_[2], *er_[2], *nrow[RN];
        double wx[RN][NF];
        int len[RN];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const size_t r = min(2 * rp + q, p.ng - 1);
            wr_[q] = p.wt + r * nc;
            er_[q] = p.ieps + r * nc;
        }
#pragma unroll
        for (int n = 0; n < RN; ++n) {
            const int4 e = nr.list[min(e0 + n, count - 1)];
            nrow[n] = p.aqsn + (size_t)e.x * nc;
            len[n] = e0 + n < count ? e.z : 0;
#pragma unroll
            for (int w = 0; w < NF; ++w)
                wx[n][w] = __ldg(p.wx + (size_t)e.x * p.wx_stride + min(e.y + w, p.nw - 1));
        }
        double2 acc[RN][2][NF];
#pragma unroll
        for (int n = 0; n < RN; ++n)
#pragma unroll
            for (int w = 0; w < NF; ++w) acc[n][0][w] = acc[n][1][w] = make_double2(0.0, 0.0);
        for (int ig = threadIdx.x; ig < nc; ig += 128) {
            double2 Q[2], wt[2];
            double wti2[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                wt[q] = __ldg(wr_[q] + ig);
                Q[q] = cmul(wt[q], __ldg(er_[q] + ig));
                wti2[q] = wt[q].y * wt[q].y;
            }
#pragma unroll
            for (int n = 0; n < RN; ++n) {
                const double2 a = __ldg(nrow[n] + ig);
                double2 A[2], Aw[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    A[q] = cmul(a, Q[q]);
                    Aw[q] = make_double2(A[q].x * wt[q].y, A[q].y * wt[q].y);
                }
#pragma unroll
                for (int w = 0; w < NF; ++w) {
                    if (w >= len[n]) break;  // the same for the whole block
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const double wr = wx[n][w] - wt[q].x;
                        const double rr = rcp_fp64(fma(wr, wr, wti2[q]));
                        acc[n][q][w].x = fma(rr, fma(A[q].x, wr, -Aw[q].y), acc[n][q][w].x);
                        acc[n][q][w].y = fma(rr, fma(A[q].y, wr, Aw[q].x), acc[n][q][w].y);
                    }
                }
            }
        }
        double v[K];
#pragma unroll
        for (int n = 0; n < RN; ++n)
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int w = 0; w < NF; ++w) {
                    v[((n * 2 + q) * NF + w) * 2] = acc[n][q][w].x;
                    v[((n * 2 + q) * NF + w) * 2 + 1] = acc[n][q][w].y;
                }
        block_reduce<K, 128>(v, red, S);
        near_epilogue<RN, NF>(p, nr, S, e0, count, rp);
        __syncthreads();
    }
}

// near_val[entry][frequency] (+)= the sum over the pass's row pairs, a warp per
// sum.
__global__ void __launch_bounds__(256) far_near_sum_kernel(FarNear nr, double2 *val) {
    if (!*nr.active) return;
    const int lane = threadIdx.x & 31, count = *nr.count * kNearFreq, pairs = nr.pairs;
    for (int e = (blockIdx.x * 256 + threadIdx.x) >> 5; e < count; e += (gridDim.x * 256) >> 5) {
        double x = 0.0, y = 0.0;
        for (int r = lane; r < pairs; r += 32) {
            const double2 v = nr.partial[(size_t)e * pairs + r];
            x += v.x;
            y += v.y;
        }
        x = warp_sum(x);
        y = warp_sum(y);
        if (lane == 0) val[e] = nr.pair0 ? cadd(val[e], make_double2(x, y)) : make_double2(x, y);
    }
}

// The strays' terms of the far pairs, FP64: blockIdx.x a segment of the list,
// blockIdx.y 4 bands, blockIdx.z up to 4 frequencies;
// part[segment][pair] (0 for near pairs).
constexpr int kOutBands = 4, kOutFreq = 4;
__global__ void __launch_bounds__(128) far_out_kernel(Problem p, const FarPlan *f, const int2 *list,
                                                      long long seg_len, int b0, int bands,
                                                      const double2 *C, const double2 *spread,
                                                      double2 *part) {
    if (!f->active) return;
    constexpr int K = kOutBands * kOutFreq * 2;
    __shared__ double red[4 * K], S[K];
    const long long a = blockIdx.x * seg_len, b = min((long long)f->n_out, a + seg_len);
    if (a >= b) return;
    const int n0 = blockIdx.y * kOutBands, w0 = blockIdx.z * kOutFreq;
    const int nc = p.nc;
    double wx[kOutBands][kOutFreq];
    bool any = false;
    unsigned far = 0;
#pragma unroll
    for (int n = 0; n < kOutBands; ++n)
#pragma unroll
        for (int w = 0; w < kOutFreq; ++w) {
            const int band = b0 + min(n0 + n, bands - 1);
            wx[n][w] = __ldg(p.wx + (size_t)band * p.wx_stride + min(w0 + w, p.nw - 1));
            if (n0 + n < bands && w0 + w < p.nw && held(spread[n0 + n]) && is_far(*f, wx[n][w])) far |= 1u << (n * kOutFreq + w);
        }
    any = far != 0;
    double2 acc[kOutBands][kOutFreq];
#pragma unroll
    for (int n = 0; n < kOutBands; ++n)
#pragma unroll
        for (int w = 0; w < kOutFreq; ++w) acc[n][w] = make_double2(0.0, 0.0);
    if (any)
        for (long long i = a + threadIdx.x; i < b; i += 128) {
            const int2 e = list[i];
            const double2 wt = __ldg(p.wt + (size_t)e.x * nc + e.y);
            const double2 Q = cmul(wt, __ldg(p.ieps + (size_t)e.x * nc + e.y));
            const double wti2 = wt.y * wt.y;
#pragma unroll
            for (int n = 0; n < kOutBands; ++n) {
                if (!((far >> (n * kOutFreq)) & ((1u << kOutFreq) - 1))) continue;
                const int k = min(n0 + n, bands - 1);
                const double2 A = cmul(cmul(__ldg(p.aqsn + (size_t)(b0 + k) * nc + e.y),
                                            C[(size_t)k * p.ng + e.x]), Q);
                const double ayw = A.y * wt.y, axw = A.x * wt.y;
#pragma unroll
                for (int w = 0; w < kOutFreq; ++w) {
                    if (!((far >> (n * kOutFreq + w)) & 1)) continue;
                    const double wr = wx[n][w] - wt.x;
                    const double rr = rcp_fp64(fma(wr, wr, wti2));
                    acc[n][w].x = fma(rr, fma(A.x, wr, -ayw), acc[n][w].x);
                    acc[n][w].y = fma(rr, fma(A.y, wr, axw), acc[n][w].y);
                }
            }
        }
    double v[K];
#pragma unroll
    for (int n = 0; n < kOutBands; ++n)
#pragma unroll
        for (int w = 0; w < kOutFreq; ++w) {
            v[(n * kOutFreq + w) * 2] = acc[n][w].x;
            v[(n * kOutFreq + w) * 2 + 1] = acc[n][w].y;
        }
    block_reduce<K, 128>(v, red, S);
    const int t = threadIdx.x, n = t / kOutFreq, w = t % kOutFreq;
    if (t < kOutBands * kOutFreq && n0 + n < bands && w0 + w < p.nw)
        part[(size_t)blockIdx.x * bands * p.nw + (size_t)(n0 + n) * p.nw + w0 + w] =
            make_double2(S[t * 2], S[t * 2 + 1]);
}

// The series of a far pair from its band's sums S1.
__device__ __forceinline__ double2 far_series(const FarPlan &f, double wx, const double2 *S1, int K) {
    const double u = (wx - f.z0) * f.inv_h;
    const double s = copysign(sqrt((u - 1.0) * (u + 1.0)), u);
    const double q = 1.0 / (u + s);
    double2 acc = make_double2(0.0, 0.0);
    for (int k = K - 1; k >= 1; --k)  // Horner in 1 / r, smallest terms first
        acc = make_double2(fma(acc.x, q, S1[k].x), fma(acc.y, q, S1[k].y));
    const double g = f.inv_h / s;
    return make_double2(g * fma(2.0 * q, acc.x, S1[0].x), g * fma(2.0 * q, acc.y, S1[0].y));
}

// Block iw < nw: that frequency's total over bands, near entries and strays;
// block nw + n: band n's total at iw = 2.  Written into the first unoccupied
// slot of the frequency, or the band's first row slot.
__global__ void __launch_bounds__(256) far_final_kernel(Problem p, const FarPlan *f, int b0, int bands,
                                                        const int4 *near, const int *place,
                                                        const double2 *near_val,
                                                        const double2 *out_part, long long seg_len,
                                                        const double2 *S1, int K, const double2 *spread,
                                                        Partials part) {
    if (!f->active) return;
    __shared__ double red[16], S[2];
    const bool band = (int)blockIdx.x >= p.nw;
    const int iw = band ? 2 : blockIdx.x;
    const int n0 = band ? blockIdx.x - p.nw : 0, n1 = band ? n0 + 1 : bands;
    const int segs = (int)((f->n_out + seg_len - 1) / seg_len);
    double v[2] = {0.0, 0.0};
    for (int n = n0 + (band ? 0 : (int)threadIdx.x); n < n1; n += 256) {
        const double wx = p.wx[(size_t)(b0 + n) * p.wx_stride + iw];
        if (!held(spread[n]) || !is_far(*f, wx)) continue;
        if (!band || threadIdx.x == 0) {
            const double2 x = far_series(*f, wx, S1 + (size_t)n * K, K);
            v[0] += x.x;
            v[1] += x.y;
        }
        for (int sg = band ? threadIdx.x : 0; sg < segs; sg += band ? 256 : 1) {
            const double2 x = out_part[(size_t)sg * bands * p.nw + (size_t)n * p.nw + iw];
            v[0] += x.x;
            v[1] += x.y;
        }
    }
    for (int l = 0; l < (band ? kNearFreq : 1); ++l) {
        const int e0 = band ? place[l * bands + n0] : 0, e1 = band ? place[l * bands + n0 + 1] : f->n_near;
        for (int e = e0 + threadIdx.x; e < e1; e += 256) {
            const int4 q = near[e];
            const int w = iw - q.y;
            if (w < 0 || w >= q.z) continue;
            v[0] += near_val[(size_t)e * kNearFreq + w].x;
            v[1] += near_val[(size_t)e * kNearFreq + w].y;
        }
    }
    block_reduce<2, 256>(v, red, S);
    if (threadIdx.x == 0) {
        if (band)
            part.n1[(long long)(b0 + n0) * part.n1_seg] = make_double2(S[0], S[1]);
        else
            part.ach[(long long)iw * part.ach_seg + part.ach_tile0] = make_double2(S[0], S[1]);
    }
}

}  // namespace

bool far_eligible(const Problem &p, int bands, bool mixed) {
    if (p.wx_stride == 0 || bands < 32 || p.ng < 16 || p.nc < 512) return false;
    const Sizes z = sizes(p, bands, mixed);
    // The series and, say, a sixth of the pairs near must leave a gain, on a
    // call long enough for the fixed launches: 3 ms of per-term work, in FP64
    // 2.2 (per term / series, ms: FP64 at estimates of 2.5 and 2.6 ms 2.88 / 2.47
    // and 2.66 / 2.24, before the bands' spread was formed 1.86 / 1.91 at 1.7; mixed at
    // 3.0, 3.0 and 3.3 ms 3.17 / 3.02, 2.93 / 2.28 and 3.39 / 3.03).  A chunk of X's
    // planes has to fit the scratch (87,000 bands), and with it the grids do.
    const double cells = (double)p.ng * p.nc;
    const double per_pair = mixed ? 2.6e-12 : 20e-12;
    // Calls whose sizes leave no gain do not plan (330 x 73 x 25601 x 2, mixed:
    // 5.2 ms through the series, 3.9 per term); FP64's per-term pairs cost up to
    // 1.6 of their 20 ps on such sizes, and the device decides.
    if (z.c0_call > (mixed ? 0.8 : 1.5) * z.pairs) return false;
    return z.c0 + 0.25 * z.pairs < 0.8 * z.pairs && cells * z.pairs * per_pair > (mixed ? 3e-3 : 2.2e-3) &&
           x_planes(z.Mp, z.Kc) <= kPassBytes / 2 && z.pairs < (1 << 20) && cells < 2e9 &&
           (z.pairs / 8 + 1) * ((p.ng + 1) / 2) < (1 << 30);  // the near kernel's tile counter
}

size_t far_bytes(const Problem &p, int bands, bool mixed) {
    return carve(sizes(p, bands, mixed), nullptr, nullptr);
}

cudaError_t far_unoccupied(const Problem &p, const Partials &part, void *ws, void *split_ws, int b0,
                           int b1, cudaStream_t s, const int **active) {
    const int bands = b1 - b0;
    const bool mixed = split_ws != nullptr;
    const Sizes z = sizes(p, bands, mixed);
    Buffers b;
    carve(z, ws, &b);
    const int *go = &b.plan->active;
    *active = go;
    const int sms = sm_count();
    far_range_kernel<<<1, 1024, 0, s>>>(p, b0, bands, b.plan);
    far_hist_kernel<<<sms * 4, 256, 0, s>>>(p, b.plan);
    const float w_near = 1.4f;
    far_plan_kernel<<<kPlanBlocks, kBins, 0, s>>>(p, b0, bands, b.plan, z.cap_out, (float)z.R, z.c0_call,
                                                  w_near, z.near_least, mixed ? 16.f : 2.f);
    const int band_warps = ceil_div(bands, 8);
    far_coeff_kernel<<<sms * 4, 256, 0, s>>>(p, b0, bands, b.C, b.plan, part.err);
    count_launch(4);
    // The spread of each band, a pass per group of rows and slab of chunks that
    // `sx`, `sy` and `res` hold (an x plane is 1 of 3 kCrtN).
    const int yp = ceil_div(z.gr, kCrtRowsY) * kCrtRowsY, np = ceil_div((long long)z.gm * z.gr, kCrtRowsY) * kCrtRowsY;
    const int spread_slab = (int)std::min<long long>(z.nch, 3ll * kCrtN / 4 * z.slab * (np / yp));
    cudaError_t e = cudaGetLastError();
    for (int r0 = 0; r0 < z.ngp && e == cudaSuccess; r0 += z.gr) {
        const int gr = std::min(z.gr, z.ngp - r0), rows = std::min(gr, p.ng - r0);
        const int sxc = z.x_all ? z.nch : 3 * kCrtN * z.slab, slab = std::min(spread_slab, sxc);
        for (int c0 = 0; c0 < z.nch && e == cudaSuccess; c0 += slab) {
            const int nc = std::min(slab, z.nch - c0);
            float *V = reinterpret_cast<float *>(b.res);
            far_sizes_kernel<false><<<z.Mp / 8 * nc, 128, 0, s>>>(p, b.plan, b0, bands, z.Mp, z.Mp, c0, nc, z.Kc,
                                                                  b.EA, b.SA, b.sx);
            far_sizes_kernel<true><<<gr / 8 * nc, 128, 0, s>>>(p, b.plan, r0, rows, gr, z.ngp, c0, nc, z.Kc,
                                                               b.E0 + r0, b.SQ + r0, b.sy);
            e = crt_sums(b.sx, b.sy, z.Mp, yp, z.Kc, nc, V, go, part.err, s);
            far_spread_kernel<<<bands, 256, 0, s>>>(b.plan, b.C, b.EA, b.E0, b.SA, b.SQ, V, p.ng, z.ngp, r0,
                                                    rows, z.Mp, yp, c0, nc, r0 + c0 > 0, b.spread);
            count_launch(3);
        }
    }
    if (e != cudaSuccess) return e;
    far_near_count_kernel<<<band_warps, 256, 0, s>>>(p, b.plan, b0, bands, b.spread, b.place);
    far_near_scan_kernel<<<1, 1024, 0, s>>>(b.plan, bands, p.nw, b.place, z.cap_near, z.c0_call, w_near,
                                             z.near_least);
    far_near_list_kernel<<<band_warps, 256, 0, s>>>(p, b.plan, b0, bands, b.spread, b.place, b.near);
    far_count_kernel<<<p.ng, 256, 0, s>>>(p, b.plan, b.rows);
    far_scan_kernel<<<1, 1024, 0, s>>>(p.ng, b.plan, b.rows);
    far_list_kernel<<<p.ng, 256, 0, s>>>(p, b.plan, b.rows, b.out);
    far_need_kernel<<<ceil_div(bands, 256), 256, 0, s>>>(p, b.plan, b0, bands, z.K, z.bits, b.spread, b.terms);
    far_order_kernel<<<ceil_div(bands, 256), 256, 0, s>>>(b.plan, bands, b.terms, b.order);
    count_launch(8);
    e = cudaGetLastError();

    // The series, a pass per group of rows, group of terms of one level and slab
    // of chunks.
    const OzOperand X{p.aqsn + (size_t)b0 * p.nc, p.nc, true, bands};
    const size_t x_slab = x_planes(z.Mp, z.Kc) / sizeof(__nv_bfloat16) * z.slab;
    int level = -1;
    for (int r0 = 0; r0 < z.ngp && e == cudaSuccess; r0 += z.gr) {
        const int gr = std::min(z.gr, z.ngp - r0), rows = std::min(gr, p.ng - r0);
        for (int k0 = 0; k0 < z.K && e == cudaSuccess;) {
            const int l = level_of(z, k0);
            int gm = 1;
            while (gm < z.gm && k0 + gm < z.K && level_of(z, k0 + gm) == l) ++gm;
            const int N = gm * gr, Np = ceil_div(N, kCrtRowsY) * kCrtRowsY;
            for (int c0 = 0, q = 0; c0 < z.nch && e == cudaSuccess; c0 += z.slab, ++q) {
                const int nc = std::min(z.slab, z.nch - c0);
                __nv_bfloat16 *sx = b.sx + (z.x_all ? q * x_slab : 0);
                int *ex = b.EX + (size_t)c0 * z.Mp;
                if (!z.x_all || l != level)
                    e = crt_rows(X, b.order, z.Mp, p.nc, z.Kc, c0, nc, l, sx, ex, go, s);
                if (e != cudaSuccess) break;
                auto terms = [&](auto kern) {
                    kern<<<gr / 8 * nc, 128, 0, s>>>(p, b.plan, z.ngp, r0, gr, c0, nc, z.Kc, Np, k0, gm,
                                                     k0 + gm >= z.K, b.sy, b.EY, b.E0, b.state);
                };
                switch (l) {
                    case kCrtWide: terms(far_terms_kernel<kCrtWide, false>); break;
                    case 0: mixed ? terms(far_terms_kernel<0, true>) : terms(far_terms_kernel<0, false>); break;
                    case 1: mixed ? terms(far_terms_kernel<1, true>) : terms(far_terms_kernel<1, false>); break;
                    case 2: mixed ? terms(far_terms_kernel<2, true>) : terms(far_terms_kernel<2, false>); break;
                    default: mixed ? terms(far_terms_kernel<3, true>) : terms(far_terms_kernel<3, false>); break;
                }
                count_launch();
                const int *live = &b.plan->bands_at[k0];  // the most of the pass's terms
                e = crt_products(sx, b.sy, z.Mp, Np, z.Kc, nc, 0, z.Mp / kCrtRowsX, l, b.res, z.Mp, go,
                                 live, part.err, s);
                if (e == cudaSuccess)
                    e = crt_combine(b.res, ex, b.EY, 0, bands, z.Mp, N, z.Mp, Np, nc, l, c0 > 0, b.H, N, go,
                                    live, s);
            }
            level = l;
            if (e != cudaSuccess) break;
            far_fold_kernel<<<dim3(bands, gm), 256, 0, s>>>(b.plan, b.order, b.C, b.H, p.ng, r0, rows, gr, N,
                                                            k0, z.K, b.S1);
            count_launch();
            k0 += gm;
        }
    }
    if (e != cudaSuccess) return e;

    for (int p0 = 0; p0 < (p.ng + 1) / 2; p0 += z.near_rows) {
        if (p0 > 0 && (e = cudaMemsetAsync(&b.plan->next, 0, sizeof(int), s)) != cudaSuccess) return e;
        const FarNear nr{b.near, &b.plan->n_near, go, b.C, b0, p0, std::min(z.near_rows, (p.ng + 1) / 2 - p0),
                         &b.plan->next, b.near_part};
        if (mixed) {
            e = launch_near_mixed(p, part, split_ws, nr, z.cap_near, s);
            if (e != cudaSuccess) return e;
        } else {
            far_near_fp64_kernel<<<sms * 2, 128, 0, s>>>(p, nr);
            count_launch();
        }
        far_near_sum_kernel<<<sms, 256, 0, s>>>(nr, b.near_val);
        count_launch();
    }
    far_out_kernel<<<dim3(z.segs, ceil_div(bands, kOutBands), ceil_div(p.nw, kOutFreq)), 128, 0, s>>>(
        p, b.plan, b.out, z.seg_len, b0, bands, b.C, b.spread, b.out_part);
    far_final_kernel<<<p.nw + (part.n1 ? bands : 0), 256, 0, s>>>(p, b.plan, b0, bands, b.near, b.place,
                                                                  b.near_val, b.out_part, z.seg_len,
                                                                  b.S1, z.K, b.spread, part);
    count_launch(2);
    return cudaGetLastError();
}

}  // namespace gpp
