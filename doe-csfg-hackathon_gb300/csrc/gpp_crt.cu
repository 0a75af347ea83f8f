// gpp_crt.cu -- FP64-accurate complex GEMM on the tensor cores by residues
// (Ozaki, Uchino and Imamura, "Ozaki Scheme II: a GEMM-oriented emulation of
// floating-point matrix multiplication using an integer modular technique",
// 2025).
//
//  * Over a chunk of at most 512 k values every operand value x of a row is
//    written as x = N 2^(e - 57), e the row's largest exponent in the chunk
//    and N a 57-bit integer (the slices of gpp_ozaki.cu hold 56 bits);
//  * the product sum of such integers is an integer X, |X| < P / 2, fixed by
//    its residues modulo 16 pairwise coprime integers p <= 256 of product
//    P = 2^125.38 (gpp_crt.cuh): 16 products of 8-bit integers, each exact in
//    bf16 with FP32 accumulation, where the slices take 36 products of slice
//    pairs (15 integers would do for 53 bits, 6% faster, but what falls off
//    below the chunk's largest value is then more than the slices lost);
//  * complex products take the 3M form (P1 = sum xr yr, P2 = sum xi yi,
//    P3 = sum (xr + xi)(yr + yi)); re = P1 - P2 and im = P3 - P1 - P2 are
//    formed on the residues, exactly;
//  * the combining pass turns the residues of re and im into 2^128 X / P and
//    rounds X 2^(ex + ey - 114) to a double; chunks are added in FP64.
//
// So the only roundings are those of the operands (to 57 bits of the chunk's
// largest value), of each chunk's result and of the sum over chunks: at the
// production shape the band sums are off by 1e-15 where the slices' float-float
// combination left 5e-15.
//
// GB300, 1638 x 32768 over 510 bands / 510 x 1638 over 32768 columns: prepare
// 0.36 / 1.4 ms, products 1.54 / 1.87 ms (1.71 / 1.41 PFLOP/s), combine 1.0 /
// 1.1 ms; the slices took 0.4 / 1.3, 4.6 / 5.4 and 1.3 / 1.4 ms.  The products
// are bound by the tensor pipe (90% of what a library GEMM reaches).
//
// crt_gemm_kernel keeps the core-matrix operand layout and the bulk-copy /
// tcgen05.mma / TMEM pipeline of gpp_ozaki.cu and makes each block
// persistent: it walks (plane, row tile, column tile) steps with the whole
// chunk of its X rows resident in shared memory (128 x 512, loaded once per
// row tile) while Y's blocks stream through a ring.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>

#include "gpp_crt.h"
#include "gpp_crt_planes.cuh"
#include "gpp_kernels.h"
#include "gpp_umma.cuh"

namespace gpp {

namespace {

constexpr int kKcMax = 512;             // k values per chunk
constexpr int kPlanes = 3 * kCrtN;      // (re, im, re + im) x moduli, at the wide level
constexpr int kTM = 128, kTN = 256;     // tcgen05.mma M (rows of X) x N (rows of Y)
constexpr int kTK = 64;                 // k per operand block
constexpr int kKSMax = kKcMax / kTK;    // operand blocks per chunk
constexpr int kStages = 3;              // ring of Y blocks (a pair of blocks: 6 half blocks each)
constexpr unsigned kBytesA = kTM * kTK * 2, kBytesB = kTN * kTK * 2;  // 16 KB, 32 KB
constexpr size_t kSmem = (size_t)kKSMax * kBytesA + (size_t)kStages * kBytesB + 512;
constexpr int kDrain = 8;     // warps that drain TMEM (16: the same time)
constexpr int kDrainCols = kTN / (kDrain / 4);
constexpr int kThreads = 64 + 32 * kDrain;  // warp 0 loads, warp 1 issues the MMAs, the rest drain
constexpr int kTmemCols = 2 * kTN;

__constant__ CrtGroup c_group[kCrtLevels][kCrtGroups] = {GPP_CRT_GROUPS};

struct Geometry {
    int M, N, K;
    int Mp, Np;      // X's rows, and a pass's rows of Y, padded to the block tile
    int nch, Kc;     // chunks, chunk length (multiple of kTK)
    int cps, splits; // chunks per split, splits
    int slab_chunks, slab_tiles;  // chunks and row tiles of X per pass
};

// The operand planes and product residues of one pass take about 4 GB each
// at most (GPP_OZAKI_FOLD_MB overrides it, for tests): a larger product runs
// in passes over rows of Y, chunks and row tiles of X.
size_t pass_budget() {
    const char *v = getenv("GPP_OZAKI_FOLD_MB");
    const long long mb = v ? atoll(v) : 0;
    return mb > 0 ? (size_t)mb << 20 : size_t(4) << 30;
}

size_t operand_bytes(const Geometry &g) {  // per chunk
    return sizeof(__nv_bfloat16) * kPlanes * (size_t)g.Kc * (g.Mp + g.Np);
}

Geometry geometry(int M, int N, int K, int splits) {
    Geometry g;
    g.M = M;
    g.N = N;
    g.K = K;
    g.nch = std::max(1, ceil_div(K, kKcMax));
    g.Kc = ceil_div(ceil_div(std::max(K, 1), g.nch), kTK) * kTK;
    g.Mp = ceil_div(std::max(M, 1), kTM) * kTM;
    const size_t y_rows = pass_budget() / (sizeof(__nv_bfloat16) * kPlanes * (size_t)g.Kc);
    g.Np = std::min(ceil_div(std::max(N, 1), kTN), (int)std::max<size_t>(1, std::min<size_t>(y_rows / kTN, 1 << 22))) * kTN;
    g.cps = ceil_div(g.nch, std::max(1, splits));
    g.splits = ceil_div(g.nch, g.cps);
    const size_t per_tile = (size_t)kPlanes * kTM * g.Np;  // residues of one row tile and chunk
    const int tiles = g.Mp / kTM;
    const size_t per_chunk = operand_bytes(g) + per_tile * tiles;
    g.slab_chunks = (int)std::max<size_t>(1, std::min<size_t>(g.cps, pass_budget() / per_chunk));
    g.slab_tiles = (int)std::max<size_t>(
        1, std::min<size_t>(tiles, pass_budget() / (per_tile * g.slab_chunks)));
    return g;
}

struct Buffers {
    __nv_bfloat16 *sx, *sy;  // [kPlanes][rows][slab k], core-matrix blocks
    int *ex, *ey;            // [slab chunks][rows]
    unsigned char *res;      // [slab chunks][kPlanes][slab rows][Np]: residues + 128
};

size_t carve(const Geometry &g, void *ws, Buffers *b) {
    char *w = static_cast<char *>(ws);
    size_t off = 0;
    auto take = [&](size_t n) {
        char *p = w + off;
        off = align_up(off + n);
        return p;
    };
    Buffers o;
    const size_t plane = sizeof(__nv_bfloat16) * kPlanes * (size_t)g.slab_chunks * g.Kc;
    o.sx = reinterpret_cast<__nv_bfloat16 *>(take(plane * g.Mp));
    o.sy = reinterpret_cast<__nv_bfloat16 *>(take(plane * g.Np));
    o.ex = reinterpret_cast<int *>(take(sizeof(int) * (size_t)g.slab_chunks * g.Mp));
    o.ey = reinterpret_cast<int *>(take(sizeof(int) * (size_t)g.slab_chunks * g.Np));
    o.res = reinterpret_cast<unsigned char *>(
        take((size_t)g.slab_chunks * kPlanes * ((size_t)g.slab_tiles * kTM) * g.Np));
    if (b) *b = o;
    return off;
}

__device__ __forceinline__ double2 operand_at(const OzOperand &z, int l, int k) {
    return __ldg(z.kfast ? z.z + (size_t)l * z.ld + k : z.z + (size_t)k * z.ld + l);
}
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}

struct PrepOperand {
    OzOperand z;
    int Lp, R;           // padded rows, rows per operand block
    __nv_bfloat16 *out;
    int *E;
    const int *order;    // row l is order[l] of z (null: l)
};

// Exponents and residue planes of chunks [c0, c0 + nc): blocks [0, x blocks)
// serve X, the rest Y.  A block stages 8 rows x one chunk in shared memory
// (each value read once, 128 contiguous bytes or more at a time), takes each
// row's largest exponent, and writes the residues of (re, im, re + im) to
// every modulus as bf16: a thread per 8 consecutive k of a row, so that a
// plane gets whole 16-byte core-matrix rows and a warp 512 contiguous bytes.
// Layout of a plane, in memory order: row tile (R rows), k step (kTK), row
// group of 8, k-core of 8, row, k -- the no-swizzle K-major core-matrix layout
// of tcgen05.mma, one contiguous block per (row tile, k step).
// Bound by its writes (6 n bytes per complex value) and the FP32 pipe.
__global__ void __launch_bounds__(256, 2) crt_prep_kernel(PrepOperand X, PrepOperand Y, int xblocks,
                                                          int K, int Kc, int c0, int nc, int nmod,
                                                          int bits, const int *go) {
    if (go && !*go) return;
    extern __shared__ __align__(16) double2 stage[];  // [8][Kc + 1]
    __shared__ unsigned long long red[8][8];
    __shared__ int exps[8];
    const bool isx = (int)blockIdx.x < xblocks;
    const PrepOperand &o = isx ? X : Y;
    const int b = isx ? blockIdx.x : blockIdx.x - xblocks;
    const int groups = o.Lp / 8;
    const int l0 = (b % groups) * 8, c = b / groups;
    const int kb = (c0 + c) * Kc, kn = min(Kc, K - kb);
    const int pitch = Kc + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const OzOperand z = o.z;

    unsigned long long mx = 0;
    if (z.kfast) {  // a warp per row
        const int l = l0 + warp;
        const int at = o.order && l < z.L ? o.order[l] : l;
#pragma unroll 4
        for (int k = lane; k < Kc; k += 32) {
            const double2 v =
                l < z.L && k < kn ? operand_at(z, at, kb + k) : make_double2(0.0, 0.0);
            stage[warp * pitch + k] = v;
            mx = max(mx, max(abs_bits(v.x), abs_bits(v.y)));
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, s));
        if (lane == 0) exps[warp] = crt_exponent(mx);
        __syncthreads();
    } else {  // lanes along the 8 rows, 4 k per warp
        const int r = lane & 7, l = l0 + r;
        const int at = o.order && l < z.L ? o.order[l] : l;
#pragma unroll 4
        for (int k = warp * 4 + (lane >> 3); k < Kc; k += 32) {
            const double2 v =
                l < z.L && k < kn ? operand_at(z, at, kb + k) : make_double2(0.0, 0.0);
            stage[r * pitch + k] = v;
            mx = max(mx, max(abs_bits(v.x), abs_bits(v.y)));
        }
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        if (lane < 8) red[warp][lane] = mx;
        __syncthreads();
        if (threadIdx.x < 8) {
#pragma unroll
            for (int w = 1; w < 8; ++w) mx = max(mx, red[w][threadIdx.x]);
            exps[threadIdx.x] = crt_exponent(mx);
        }
        __syncthreads();
    }
    if (threadIdx.x < 8) o.E[(size_t)c * o.Lp + l0 + threadIdx.x] = exps[threadIdx.x];

    const int row = threadIdx.x & 7;
    const int e = exps[row];
    const int ksteps = nc * (Kc / kTK);
    const size_t plane = (size_t)o.Lp * ksteps * kTK;
    const size_t base = ((size_t)(l0 / o.R) * ksteps * (o.R / 8) + (size_t)(l0 % o.R) / 8) * 512 + row * 8;
    for (int kg = threadIdx.x >> 3; kg < Kc / 8; kg += 32) {
        float2 dr[4][4], di[4][4];  // [pair of k][digit]
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            float a[4], bb[4], cr[4], ci[4];
            const double2 v0 = stage[row * pitch + kg * 8 + 2 * t];
            const double2 v1 = stage[row * pitch + kg * 8 + 2 * t + 1];
            crt_digits(oz_fixed_point(v0.x, e, bits), a);
            crt_digits(oz_fixed_point(v1.x, e, bits), bb);
            crt_digits(oz_fixed_point(v0.y, e, bits), cr);
            crt_digits(oz_fixed_point(v1.y, e, bits), ci);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                dr[t][k] = f2(a[k], bb[k]);
                di[t][k] = f2(cr[k], ci[k]);
            }
        }
        const int ks = c * (Kc / kTK) + (kg >> 3);
        __nv_bfloat16 *w = o.out + base + (size_t)ks * (o.R / 8) * 512 + (kg & 7) * 64;
        crt_store_residues<4, 4>(dr, di, nmod, w, plane);
    }
}

// The steps of one block (or pair: a row tile is then two): planes q in groups of `gq`, the (plane, row tile,
// column tile) steps of a group in order, each block a contiguous run of them
// (rotated from group to group, so that the runs' rounding evens out).
// Consecutive steps of a row tile share X's rows in shared memory, and the
// blocks in flight work on a few planes, whose operands fit in L2.
struct Walk {
    int Q, MT, NT, gq, grid;
    unsigned unit;  // this block, or pair of blocks
    int g = 0;
    long long t = 0, end = 0;
    int q0 = 0, q = 0, mt = 0, nt = 0;
    bool first = false;  // this step starts a row tile's run (X's rows change)
    __device__ __forceinline__ bool open_group() {
        for (; g * gq < Q; ++g) {
            q0 = g * gq;
            const long long steps = (long long)min(gq, Q - q0) * MT * NT;
            const long long j = (long long)((unit + (unsigned)g * 61u) % (unsigned)grid);
            t = j * steps / grid;
            end = (j + 1) * steps / grid;
            if (t < end) return true;
        }
        return false;
    }
    __device__ __forceinline__ void decode() {
        const int per = MT * NT;
        q = q0 + (int)(t / per);
        const int r = (int)(t % per);
        mt = r / NT;
        nt = r % NT;
    }
    __device__ __forceinline__ bool start() {
        if (!open_group()) return false;
        decode();
        first = true;
        return true;
    }
    // Whether the next step leaves this row tile's run.
    __device__ __forceinline__ bool last() const { return t + 1 == end || nt + 1 == NT; }
    __device__ __forceinline__ bool next() {
        if (++t == end) {
            ++g;
            return start();
        }
        first = false;
        if (++nt == NT) {
            nt = 0;
            first = true;
            if (++mt == MT) {
                mt = 0;
                ++q;
            }
        }
        return true;
    }
};

// Residues of the products: plane q = c (3 nmod) + (3M plane, modulus) of the
// pass's chunks, rows [128 mt0, + 128 MT) of X against every row of Y; the
// byte stored is the symmetric residue + 128, at res[(q Ms + row) Np + col].
// Warp 0 (one thread) loads: X's blocks of a row tile into kKSMax resident
// slots, each as soon as the MMAs of the previous run's last step released
// it, and Y's blocks through a ring, all by 1-D bulk copies onto mbarriers;
// warp 1 issues four K = 16 tcgen05.mma per block into one of two TMEM
// accumulators; warps 2-9 drain a finished accumulator (a warp's 32 lanes x
// 128 columns), reduce the exact FP32 sums modulo p on the FP32 pipe and store
// bytes, 32 in one store per thread.  Warp 1 waits as a whole and one elected
// lane issues, so that addresses and descriptors stay in uniform registers:
// run by one thread, the loop's own latency (4 MMAs 280 cycles, the commits 130,
// two waits 170) kept the tensor pipe at 53%; now 1073 -> 750 cycles a block.
// CG = 2: a pair of blocks takes two row tiles (cta_group::2, M = 256); each
// holds its own 128 rows of X and half of Y's rows, block 0 issues for both,
// and block 1's warp 1 passes on to block 0's barriers what has landed in its
// own shared memory.
// RAW: one plane of each operand, and the sums themselves as floats at
// [(q Ms + row) Np + col] of the output.
// Every wait is bounded; a block that gives up records kErrPipelineTimeout,
// lets its copies and MMAs finish and frees its TMEM.
template <int CG, bool RAW>
__global__ void __launch_bounds__(kThreads, 1)
crt_gemm_kernel(const __nv_bfloat16 *__restrict__ SX, const __nv_bfloat16 *__restrict__ SY, int Mp,
                int Np, int KS, int nc, int mt0, int MT, int gq, void *__restrict__ res,
                int Ms, int nmod, const int *go, const int *rows, int *err) {
    if (go && !*go) return;
    if (rows) MT = min(MT, (*rows + kTM - 1) / kTM);
    if (MT <= 0) return;
    constexpr int STAGES = kStages * CG;
    constexpr unsigned BYTES_B = kBytesB / CG, IDESC = umma_idesc(kTM * CG, kTN);
    const int rank = CG == 2 ? cluster_rank() : 0;
    const int planes = RAW ? 1 : 3 * nmod;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *sA = smem;
    unsigned char *sB = smem + (size_t)kKSMax * kBytesA;
    unsigned long long *bars = reinterpret_cast<unsigned long long *>(sB + (size_t)kStages * kBytesB);
    unsigned long long *full = bars, *empty = full + STAGES;
    unsigned long long *afull = empty + STAGES, *aempty = afull + kKSMax;
    unsigned long long *accfull = aempty + kKSMax, *accempty = accfull + 2;
    unsigned *tmem_slot = reinterpret_cast<unsigned *>(accempty + 2);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
    __shared__ int issued_a, issued_b, waited_a, waited_b;
    volatile int *abort = abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ksteps = nc * KS;
    Walk w;
    w.Q = nc * planes;
    w.MT = (MT + CG - 1) / CG;
    w.NT = Np / kTN;
    w.gq = gq;
    w.grid = gridDim.x / CG;
    w.unit = blockIdx.x / CG;

    if (tid == 0) {
        // Block 0 of a pair also waits for the other block's copies.
        const int arrivals = CG == 2 && rank == 0 ? 2 : 1;
        for (int s = 0; s < STAGES; ++s) {
            bar_init(&full[s], arrivals);
            bar_init(&empty[s], 1);
        }
        for (int s = 0; s < kKSMax; ++s) {
            bar_init(&afull[s], arrivals);
            bar_init(&aempty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            bar_init(&accfull[a], 1);
            bar_init(&accempty[a], kDrain * CG);
        }
        *abort_flag = 0;
        issued_a = issued_b = waited_a = waited_b = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             smem_addr(tmem_slot)),
                         "r"(kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             smem_addr(tmem_slot)),
                         "r"(kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (CG == 2) cluster_sync();  // both blocks' barriers are there
    tc_fence_after();
    const unsigned tmem = *tmem_slot;

    auto commit = [](unsigned long long *bar) {
        if constexpr (CG == 2)
            umma_commit_pair(bar);
        else
            umma_commit(bar);
    };
    if (warp == 0) {
        if (lane == 0) {  // producer
            const size_t xplane = (size_t)Mp * ksteps * kTK, yplane = (size_t)Np * ksteps * kTK;
            int run = -1, nb = 0;  // row-tile runs and Y blocks so far
            bool ok = true;
            for (bool more = w.start(); ok && more; more = w.next()) {
                const int c = w.q / planes, pl = w.q % planes;
                const __nv_bfloat16 *a = SX + pl * xplane +
                                         ((size_t)(mt0 + min(w.mt * CG + rank, MT - 1)) * ksteps + (size_t)c * KS) * (kTM * kTK);
                const __nv_bfloat16 *b =
                    SY + pl * yplane + ((size_t)w.nt * ksteps + (size_t)c * KS) * (kTN * kTK) +
                    rank * (BYTES_B / sizeof(__nv_bfloat16));
                if (w.first) ++run;
                for (int s = 0; s < KS; ++s) {
                    if (w.first) {
                        if (run > 0 && !bar_wait(&aempty[s], (run - 1) & 1, abort)) { ok = false; break; }
                        bar_expect_tx(&afull[s], kBytesA);
                        bulk_g2s(sA + (size_t)s * kBytesA, a + (size_t)s * (kTM * kTK), kBytesA, &afull[s]);
                        ++issued_a;
                    }
                    const int st = nb % STAGES;
                    if (nb >= STAGES && !bar_wait(&empty[st], (nb / STAGES - 1) & 1, abort)) {
                        ok = false;
                        break;
                    }
                    bar_expect_tx(&full[st], BYTES_B);
                    bulk_g2s(sB + (size_t)st * BYTES_B, b + (size_t)s * (kTN * kTK), BYTES_B, &full[st]);
                    ++nb;
                }
            }
            issued_b = nb;
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 1) {  // tells block 0 what has landed here
            int run = -1, nb = 0;
            bool ok = true;
            for (bool more = w.start(); ok && more; more = w.next()) {
                if (w.first) ++run;
                for (int s = 0; s < KS; ++s) {
                    if (w.first) {
                        if (!bar_wait(&afull[s], run & 1, abort)) { ok = false; break; }
                        bar_arrive_leader(&afull[s]);
                        ++waited_a;
                    }
                    const int st = nb % STAGES;
                    if (!bar_wait(&full[st], (nb / STAGES) & 1, abort)) { ok = false; break; }
                    bar_arrive_leader(&full[st]);
                    ++nb;
                }
            }
            waited_b = nb;
        } else if (rank == 0) {  // MMA issuer: the warp waits, one lane issues
            const bool one = elect_one();
            const unsigned sa0 = smem_addr(sA), sb0 = smem_addr(sB);
            int run = -1, nb = 0, st = 0, G = 0;
            unsigned phase = 0;
            bool ok = true;
            for (bool more = w.start(); ok && more; more = w.next(), ++G) {
                if (w.first) ++run;
                const bool last = w.last();
                const int acc = G & 1;
                if (G >= 2 && !__all_sync(~0u, bar_wait(&accempty[acc], ((G >> 1) - 1) & 1, abort))) break;
                tc_fence_after();
                for (int s = 0; s < KS; ++s) {
                    if (w.first) {
                        ok = __all_sync(~0u, bar_wait(&afull[s], run & 1, abort));
                        if (!ok) break;
                        if (one) ++waited_a;
                    }
                    ok = __all_sync(~0u, bar_wait(&full[st], phase, abort));
                    if (!ok) break;
                    const unsigned long long da = umma_desc(sa0 + (unsigned)s * kBytesA, 128, 1024),
                                             db = umma_desc(sb0 + (unsigned)st * BYTES_B, 128, 1024);
                    if (one) {
#pragma unroll
                        for (int k16 = 0; k16 < kTK / 16; ++k16) {  // 256 bytes on in both
                            const unsigned add = !(s == 0 && k16 == 0);
                            if constexpr (CG == 2)
                                umma_bf16_pair(tmem + acc * kTN, da + k16 * 16, db + k16 * 16, IDESC, add);
                            else
                                umma_bf16(tmem + acc * kTN, da + k16 * 16, db + k16 * 16, IDESC, add);
                        }
                        commit(&empty[st]);
                        if (last) commit(&aempty[s]);
                        if (s == KS - 1) commit(&accfull[acc]);
                    }
                    __syncwarp();
                    ++nb;
                    if (++st == STAGES) {
                        st = 0;
                        phase ^= 1;
                    }
                }
            }
            if (one) waited_b = nb;
        }
    } else {  // epilogue: TMEM lanes 32 (warp % 4) .., columns kDrainCols ((warp - 2) / 4) ..
        const int quarter = warp & 3, group = (warp - 2) >> 2;
        int G = 0;
        for (bool more = w.start(); more; more = w.next(), ++G) {
            const int acc = G & 1;
            if (!bar_wait(&accfull[acc], (G >> 1) & 1, abort)) break;
            tc_fence_after();
            const CrtMod m = RAW ? CrtMod{} : c_crt_mod[(w.q % planes) % nmod];
            const int tile = w.mt * CG + rank;  // the pair's second may be past the end
            const size_t at = ((size_t)w.q * Ms + (size_t)tile * kTM + quarter * 32 + lane) * Np +
                              (size_t)w.nt * kTN + group * kDrainCols;
            const unsigned ta = tmem + ((unsigned)(quarter * 32) << 16) + acc * kTN + group * kDrainCols;
#pragma unroll 1
            for (int cc = 0; cc < kDrainCols; cc += 32) {
                float v[32];
                tmem_ld32(ta + cc, v);
                if constexpr (RAW) {
                    float4 *o = reinterpret_cast<float4 *>(static_cast<float *>(res) + at + cc);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (tile < MT) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    continue;
                }
                unsigned char *o = static_cast<unsigned char *>(res) + at;
                unsigned word[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    // r + 128 (mod 256) in the low byte of r + 2^23 + 128's bits.
                    const float2 off = f2(8388608.0f + 128.0f, 8388608.0f + 128.0f);
                    const float2 x = f2add(crt_reduce2(f2(v[4 * j], v[4 * j + 1]), m.p, m.inv), off);
                    const float2 y = f2add(crt_reduce2(f2(v[4 * j + 2], v[4 * j + 3]), m.p, m.inv), off);
                    const unsigned lo = __byte_perm(__float_as_uint(x.x), __float_as_uint(x.y), 0x0040);
                    const unsigned hi = __byte_perm(__float_as_uint(y.x), __float_as_uint(y.y), 0x0040);
                    word[j] = __byte_perm(lo, hi, 0x5410);
                }
                if (tile < MT)  // 32 bytes per thread in one store
                    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + cc),
                                 "r"(word[0]), "r"(word[1]), "r"(word[2]), "r"(word[3]), "r"(word[4]),
                                 "r"(word[5]), "r"(word[6]), "r"(word[7])
                                 : "memory");
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if constexpr (CG == 2)
                    bar_arrive_leader(&accempty[acc]);
                else
                    bar_arrive(&accempty[acc]);
            }
        }
    }

    __syncthreads();
    if (*abort && tid == 0) {
        atomicOr(err, kErrPipelineTimeout);
        // Let the copies still in flight land and the issued MMAs finish.
        auto settle = [&](unsigned long long *bar, unsigned parity) {
            int spin = 0;
            while (!bar_try_wait(bar, parity) && ++spin < kWaitLimit) {
            }
        };
        for (int t = waited_b; t < issued_b; ++t)
            settle(&full[t % STAGES], (unsigned)((t / STAGES) & 1));
        for (int t = waited_a; t < issued_a; ++t)
            settle(&afull[t % KS], (unsigned)((t / KS) & 1));
        if (waited_b > 0)
            settle(&empty[(waited_b - 1) % STAGES], (unsigned)(((waited_b - 1) / STAGES) & 1));
    }
    tc_fence_before();
    __syncthreads();
    // Neither block goes while the other's MMAs or arrivals may reach it.
    if constexpr (CG == 2) cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        if constexpr (CG == 1)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                         "r"(kTmemCols)
                         : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                         "r"(kTmemCols)
                         : "memory");
    }
}

// Out (= or +=) the pass's chunks: a thread per row and 4 consecutive
// columns reads the 3 n residue words of a chunk, forms the residues of re and
// im for each column, their sum of fractions (integer multiply-adds) and
// X 2^(ex + ey - 2 bits), and adds it to the running FP64 result, chunk by chunk.
// Bound by integer issue.
template <int L>
__global__ void __launch_bounds__(128, 5) crt_combine_kernel(const unsigned char *res, const int *EX,
                                                             const int *EY, int row0, int rows,
                                                             int Ms, int N, int Mp, int Np, int nc,
                                                             int accumulate, double2 *Out,
                                                             long long out_ld, const int *go,
                                                             const int *live) {
    if (go && !*go) return;
    if (live) rows = min(rows, *live);
    constexpr int NM = kCrtLevel[L].n, PLANES = 3 * NM, GROUPS = (NM + 1) / 2;
    const unsigned quads = (N + 3) / 4;
    const long long n = (long long)rows * quads;
    const size_t plane = (size_t)Ms * Np;
    for (long long t = (long long)blockIdx.x * 128 + threadIdx.x; t < n;
         t += (long long)gridDim.x * 128) {
        int r, col0;
        if (n < (1ll << 31)) {
            r = (int)((unsigned)t / quads);
            col0 = (int)((unsigned)t % quads) * 4;
        } else {
            r = (int)(t / quads);
            col0 = (int)(t % quads) * 4;
        }
        double2 *out = Out + (long long)(row0 + r) * out_ld + col0;
        double2 acc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            acc[j] = accumulate && col0 + j < N ? out[j] : make_double2(0.0, 0.0);
        for (int c = 0; c < nc; ++c) {
            const unsigned char *f = res + (size_t)c * PLANES * plane + (size_t)r * Np + col0;
            unsigned u[PLANES];
#pragma unroll
            for (int q = 0; q < PLANES; ++q)
                u[q] = __ldg(reinterpret_cast<const unsigned *>(f + q * plane));
            const int ex = __ldg(EX + (size_t)c * Mp + row0 + r);
            const int4 ey = __ldg(reinterpret_cast<const int4 *>(EY + (size_t)c * Np + col0));
            // Not unrolled: the residue words take up to 48 registers, and one column's
            // state at a time leaves room for five blocks per SM.
#pragma unroll 1
            for (int j = 0; j < 4; ++j) {
                CrtSum re, im;
                const unsigned sel = 0x4440 + j;
#pragma unroll
                for (int k = 0; k < GROUPS; ++k) {
                    int rr[2] = {0, 0}, ri[2] = {0, 0};
#pragma unroll
                    for (int h = 0; h < 2 && 2 * k + h < NM; ++h) {
                        const int i = 2 * k + h;
                        const int a = __byte_perm(u[i], 0, sel);
                        const int b = __byte_perm(u[NM + i], 0, sel);
                        rr[h] = a - b;                                      // r1 - r2
                        ri[h] = (int)__byte_perm(u[2 * NM + i], 0, sel) - a - b;  // r3 - r1 - r2 - 128
                    }
                    re.add<0>(rr[0], rr[1], c_group[L][k]);
                    im.add<-128>(ri[0], ri[1], c_group[L][k]);
                }
                const int eyj = j == 0 ? ey.x : j == 1 ? ey.y : j == 2 ? ey.z : ey.w;
                double2 v;
                if (ex >= kExpNonFinite || eyj >= kExpNonFinite)
                    v.x = v.y = __longlong_as_double(0x7FF8000000000000ll);
                else
                    v = make_double2(crt_value<L>(re, ex + eyj - 2 * kCrtLevel[L].bits),
                                     crt_value<L>(im, ex + eyj - 2 * kCrtLevel[L].bits));
                if (c == 0 && !accumulate && nc == 1) {
                    if (col0 + j < N) out[j] = v;
                    continue;
                }
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (m == j) acc[m] = c == 0 && !accumulate ? v : cadd(acc[m], v);
            }
        }
        if (nc == 1 && !accumulate) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (col0 + j < N) out[j] = acc[j];
    }
}

// Pairs of blocks (cta_group::2): each SM then reads half of Y's block for the
// same products.  16384 columns, 510 bands, 1 / 3 / 5 / 7 / 13 row tiles:
// single blocks 0.128 / 0.263 / 0.407 / 0.543 / 0.976 ms, pairs 0.138 / 0.240 /
// 0.328 / 0.432 / 0.726 (an odd row tile leaves half of a pair idle).
bool gemm_pairs(int tiles) { return tiles >= 2; }

// A launch of `grid` blocks (cg 1) or pairs of blocks (cg 2, a cluster each).
struct GemmLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute pair = {};
    GemmLaunch(int cg, int grid, cudaStream_t s) {
        cfg.gridDim = dim3(grid * cg);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = kSmem;
        cfg.stream = s;
        pair.id = cudaLaunchAttributeClusterDimension;
        pair.val.clusterDim.x = 2;
        pair.val.clusterDim.y = pair.val.clusterDim.z = 1;
        cfg.attrs = &pair;
        cfg.numAttrs = cg == 2 ? 1 : 0;
    }
    GemmLaunch(const GemmLaunch &) = delete;
};

// Pairs the device holds at once, one persistent pair each.
int pair_count() {
    static std::atomic<int> count[256] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    int n = count[dev & 255].load(std::memory_order_acquire);
    if (n == 0) {
        GemmLaunch l(2, std::max(1, sm_count() / 2), nullptr);
        if (cudaOccupancyMaxActiveClusters(&n, crt_gemm_kernel<2, false>, &l.cfg) != cudaSuccess) return 0;
        count[dev & 255].store(n, std::memory_order_release);
    }
    return n;
}

cudaError_t configure() {
    static std::atomic<bool> configured[256] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || configured[dev & 255].load(std::memory_order_acquire)) return e;
    for (auto kern : {crt_gemm_kernel<1, false>, crt_gemm_kernel<2, false>, crt_gemm_kernel<1, true>,
                      crt_gemm_kernel<2, true>})
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(crt_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double2) * 8 * (kKcMax + 1)));
    if (e == cudaSuccess) configured[dev & 255].store(true, std::memory_order_release);
    return e;
}

void launch_prep(const PrepOperand &px, const PrepOperand &py, int xblocks, int yblocks, int K,
                 int Kc, int c0, int nc, int level, const int *go, cudaStream_t s) {
    crt_prep_kernel<<<xblocks + yblocks, 256, sizeof(double2) * 8 * (Kc + 1), s>>>(
        px, py, xblocks, K, Kc, c0, nc, kCrtLevel[level].n, kCrtLevel[level].bits, go);
}

}  // namespace

cudaError_t crt_rows(const OzOperand &X, const int *order, int Mp, int K, int Kc, int c0, int nc,
                     int level, void *sx, int *ex, const int *go, cudaStream_t s) {
    cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    const PrepOperand px{X, Mp, kTM, static_cast<__nv_bfloat16 *>(sx), ex, order};
    launch_prep(px, px, Mp / 8 * nc, 0, K, Kc, c0, nc, level, go, s);
    count_launch();
    return cudaGetLastError();
}

namespace {
template <bool RAW>
cudaError_t products(const void *sx, const void *sy, int Mp, int Np, int Kc, int nc, int mt0, int tiles,
                     int nmod, void *res, int Ms, const int *go, const int *rows, int *err,
                     cudaStream_t s) {
    cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    const int planes = RAW ? 1 : 3 * nmod, ntiles = Np / kTN;
    const int cg = gemm_pairs(tiles) ? 2 : 1, units = ceil_div(tiles, cg);  // row tiles, or pairs
    const int fit = cg == 2 ? pair_count() : sm_count();
    if (fit <= 0) return cudaErrorUnknown;
    const int grid = (int)std::min<long long>(fit, (long long)nc * planes * units * ntiles);
    // Planes in flight: enough that every block has a step, with their
    // operands within about 80 MB of L2.
    const size_t plane = sizeof(__nv_bfloat16) * (size_t)Kc * (Mp + Np);
    const int gq = std::max(ceil_div(grid, (long long)units * ntiles),
                            std::min(ceil_div(grid, units), (int)((size_t(80) << 20) / plane)));
    const __nv_bfloat16 *x = static_cast<const __nv_bfloat16 *>(sx),
                        *y = static_cast<const __nv_bfloat16 *>(sy);
    GemmLaunch l(cg, grid, s);
    e = cudaLaunchKernelEx(&l.cfg, cg == 2 ? crt_gemm_kernel<2, RAW> : crt_gemm_kernel<1, RAW>, x, y, Mp,
                           Np, Kc / kTK, nc, mt0, tiles, gq, res, Ms, nmod, go, rows, err);
    if (e != cudaSuccess) return e;
    count_launch();
    return cudaGetLastError();
}
}  // namespace

cudaError_t crt_products(const void *sx, const void *sy, int Mp, int Np, int Kc, int nc, int mt0,
                         int tiles, int level, unsigned char *res, int Ms, const int *go,
                         const int *rows, int *err, cudaStream_t s) {
    return products<false>(sx, sy, Mp, Np, Kc, nc, mt0, tiles, kCrtLevel[level].n, res, Ms, go, rows,
                           err, s);
}

cudaError_t crt_sums(const void *sx, const void *sy, int Mp, int Np, int Kc, int nc, float *out,
                     const int *go, int *err, cudaStream_t s) {
    return products<true>(sx, sy, Mp, Np, Kc, nc, 0, Mp / kTM, 1, out, Mp, go, nullptr, err, s);
}

cudaError_t crt_combine(const unsigned char *res, const int *ex, const int *ey, int row0, int rows,
                        int Ms, int N, int Mp, int Np, int nc, int level, bool accumulate,
                        double2 *Out, long long out_ld, const int *go, const int *live,
                        cudaStream_t s) {
    const long long want = ((long long)rows * ceil_div(N, 4) + 127) / 128;
    const int grid = (int)std::min<long long>(want, (long long)sm_count() * 32);
    auto launch = [&](auto kern) {
        kern<<<grid, 128, 0, s>>>(res, ex, ey, row0, rows, Ms, N, Mp, Np, nc, accumulate, Out, out_ld,
                                  go, live);
    };
    switch (level) {
        case 0: launch(crt_combine_kernel<0>); break;
        case 1: launch(crt_combine_kernel<1>); break;
        case 2: launch(crt_combine_kernel<2>); break;
        case 3: launch(crt_combine_kernel<3>); break;
        default: launch(crt_combine_kernel<kCrtWide>); break;
    }
    count_launch();
    return cudaGetLastError();
}

size_t crt_bytes(int M, int N, int K, int splits) {
    return carve(geometry(M, N, K, splits), nullptr, nullptr);
}

int crt_splits(int K, int splits) { return geometry(1, 1, K, splits).splits; }

cudaError_t crt_zgemm(const OzOperand &X, const OzOperand &Y, int M, int N, int K, int splits,
                      double2 *Out, long long out_ld, long long split_stride, void *ws, int *err,
                      cudaStream_t s, cudaEvent_t after_slices) {
    if (M <= 0 || N <= 0) return cudaSuccess;
    const Geometry g = geometry(M, N, K, splits);
    Buffers b;
    carve(g, ws, &b);
    cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    const int mtiles = g.Mp / kTM, Ms = g.slab_tiles * kTM;
    for (int z = 0; z < g.splits; ++z) {
        const int zc0 = z * g.cps, zc1 = std::min(g.nch, zc0 + g.cps);
        for (int c0 = zc0; c0 < zc1; c0 += g.slab_chunks) {
            const int nc = std::min(g.slab_chunks, zc1 - c0);
            for (int n0 = 0; n0 < N; n0 += g.Np) {
                OzOperand Yn = Y;
                Yn.z += (long long)n0 * (Y.kfast ? Y.ld : 1);
                Yn.L = std::min(N - n0, g.Np);
                const int Np = ceil_div(Yn.L, kTN) * kTN;
                const PrepOperand px{X, g.Mp, kTM, b.sx, b.ex, nullptr},
                    py{Yn, Np, kTN, b.sy, b.ey, nullptr};
                // X's planes serve every pass over rows of Y.
                launch_prep(px, py, n0 == 0 ? g.Mp / 8 * nc : 0, Np / 8 * nc, K, g.Kc, c0, nc,
                            kCrtWide, nullptr, s);
                count_launch();
                if (after_slices && z == 0 && c0 == 0 && n0 == 0) {
                    e = cudaEventRecord(after_slices, s);
                    if (e != cudaSuccess) return e;
                }
                for (int mt0 = 0; mt0 < mtiles; mt0 += g.slab_tiles) {
                    const int tiles = std::min(g.slab_tiles, mtiles - mt0);
                    const int row0 = mt0 * kTM, rows = std::min(M - row0, tiles * kTM);
                    e = crt_products(b.sx, b.sy, g.Mp, Np, g.Kc, nc, mt0, tiles, kCrtWide, b.res, Ms,
                                     nullptr, nullptr, err, s);
                    if (e == cudaSuccess && rows > 0)
                        e = crt_combine(b.res, b.ex, b.ey, row0, rows, Ms, Yn.L, g.Mp, Np, nc, kCrtWide,
                                        c0 > zc0, Out + z * split_stride + n0, out_ld, nullptr, nullptr, s);
                    if (e != cudaSuccess) return e;
                }
            }
        }
    }
    return cudaGetLastError();
}

}  // namespace gpp
