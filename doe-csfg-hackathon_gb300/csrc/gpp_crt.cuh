// gpp_crt.cuh -- the residue arithmetic of gpp_crt.cu, host and device: a
// fixed-point operand value as residues of up to 16 moduli, and an exact integer
// from the residues of a product sum (Chinese remainder theorem).
#pragma once

#include <cuda_runtime.h>

#include "gpp_df2.cuh"
#include "gpp_ozaki_split.cuh"

namespace gpp {

// The 16 largest pairwise coprime integers up to 256 (GPP_CRT_MODULI and 193);
// the product of the first 15 is 2^117.78, of all 2^125.38.  Symmetric
// residues |r| <= p / 2 <= 128 are integers that bf16 holds exactly, and a sum
// of 512 products of two of them is at most 2^23, which FP32 accumulation adds
// exactly.
constexpr int kCrtN = 16;
#define GPP_CRT_MODULI \
    256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197
constexpr int kCrtModuli[kCrtN] = {GPP_CRT_MODULI, 193};
// Levels of precision: the first n moduli with operands of `bits` bits,
// 2 512 2^(2 bits) < P / 2 for the product P of the n.  The last, wide one
// stands for FP64 operands: four bits more than a double's 53 for what falls
// off below a chunk's largest value.
constexpr int kCrtLevels = 5, kCrtWide = 4, kCrtWideBits = 57;
struct CrtLevel {
    int n, bits;
    unsigned long long pn;  // P = pn 2^pe, its top 64 bits rounded
    int pe;
    unsigned long long off_hi, off_lo;  // below
    unsigned zero;  // what a zero's rounding can leave of the 2^128: below
};
constexpr CrtLevel kCrtLevel[kCrtLevels] = {
    {15, 53, 0xDC47122BAA0C0C41ull, 54, 0xFFFFFFFFFFFFFFFFull, 0xFFFFFFFFFECC9200ull, 71000000u},
    {12, 41, 0xDF6327787D5133B8ull, 31, 0xFFFFFFFFFFFFFFFFull, 0xFFFFFB6A7F4B9E00ull, 71000000u},
    {9, 30, 0xAA977B6D2077B785ull, 8, 0xFFFFFFFFFFFFFFFCull, 0xFFA9A1B5A960FA00ull, 71000000u},
    {6, 18, 0xE06F178117000000ull, -16, 0xFFFFFFFFFDB7FD11ull, 0x05004945E2C6AA00ull, 71000000u},
    {kCrtN, kCrtWideBits, 0xA61194B2EB33153Dull, 62, 0xFFFFFFFFFFFFFFFFull, 0xFFFFFFFFFE27E800ull, 82000000u}};

// The residues of a pair of moduli (p, q) enter as t = r_p a + r_q b, with
// a = w_p q mod p q, b = w_q p mod p q and w_p = (P / p)^-1 mod p: then
// X / P = sum over the groups of t / (p q) (mod 1) for X = r mod every
// modulus, formed with E = round(2^128 / (p q)), least significant word first.
// A level's off is -512 sum (a + b) E mod 2^128: t is offset by 512 (a + b) to
// be positive.  Its zero is half a unit of each E times the largest residues,
// sum 382 (a + b) / 2, rounded up.
constexpr int kCrtGroups = 8;
struct CrtGroup {
    unsigned a, b, E[4];
};
#define GPP_CRT_GROUPS \
    {{57375u, 35072u, {0x01010101u, 0x01010101u, 0x01010101u, 0x00010101u}}, \
     {47941u, 45793u, {0xA0B226C6u, 0x2BC9BD16u, 0x15BEAF4Eu, 0x00010832u}}, \
     {28920u, 247u, {0xD7954FBDu, 0xC9000119u, 0x954FBCA2u, 0x000119D7u}}, \
     {32620u, 19120u, {0x317BC258u, 0x9B9BA76Cu, 0xEDD3DBC1u, 0x00012D46u}}, \
     {14755u, 14427u, {0xD9951FDCu, 0x220C9DF6u, 0x89404322u, 0x000142BEu}}, \
     {20615u, 17840u, {0x4AF518C9u, 0x79C54F61u, 0x7F7279BAu, 0x00015AB3u}}, \
     {9552u, 27008u, {0xC98E25D0u, 0xC687FEF9u, 0xEA710C29u, 0x00018F8Fu}}, \
     {91u, 0u, {0x3FACD51Eu, 0x4F44DF83u, 0x725AF6E7u, 0x014CAB88u}}}, \
    {{47175u, 54016u, {0x01010101u, 0x01010101u, 0x01010101u, 0x00010101u}}, \
     {31124u, 19228u, {0xA0B226C6u, 0x2BC9BD16u, 0x15BEAF4Eu, 0x00010832u}}, \
     {17352u, 57057u, {0xD7954FBDu, 0xC9000119u, 0x954FBCA2u, 0x000119D7u}}, \
     {10485u, 18642u, {0x317BC258u, 0x9B9BA76Cu, 0xEDD3DBC1u, 0x00012D46u}}, \
     {10215u, 49693u, {0xD9951FDCu, 0x220C9DF6u, 0x89404322u, 0x000142BEu}}, \
     {2170u, 33227u, {0x4AF518C9u, 0x79C54F61u, 0x7F7279BAu, 0x00015AB3u}}}, \
    {{19635u, 61952u, {0x01010101u, 0x01010101u, 0x01010101u, 0x00010101u}}, \
     {29869u, 55913u, {0xA0B226C6u, 0x2BC9BD16u, 0x15BEAF4Eu, 0x00010832u}}, \
     {25546u, 56810u, {0xD7954FBDu, 0xC9000119u, 0x954FBCA2u, 0x000119D7u}}, \
     {38212u, 34894u, {0x317BC258u, 0x9B9BA76Cu, 0xEDD3DBC1u, 0x00012D46u}}, \
     {161u, 0u, {0xEF3B3FB8u, 0x313011E2u, 0xB3FB8744u, 0x011E2EF3u}}}, \
    {{42585u, 37376u, {0x01010101u, 0x01010101u, 0x01010101u, 0x00010101u}}, \
     {13303u, 61479u, {0xA0B226C6u, 0x2BC9BD16u, 0x15BEAF4Eu, 0x00010832u}}, \
     {49646u, 45448u, {0xD7954FBDu, 0xC9000119u, 0x954FBCA2u, 0x000119D7u}}}, \
    {{8415u, 57344u, {0x01010101u, 0x01010101u, 0x01010101u, 0x00010101u}}, \
     {48945u, 39721u, {0xA0B226C6u, 0x2BC9BD16u, 0x15BEAF4Eu, 0x00010832u}}, \
     {32535u, 1235u, {0xD7954FBDu, 0xC9000119u, 0x954FBCA2u, 0x000119D7u}}, \
     {42872u, 55209u, {0x317BC258u, 0x9B9BA76Cu, 0xEDD3DBC1u, 0x00012D46u}}, \
     {6810u, 28625u, {0xD9951FDCu, 0x220C9DF6u, 0x89404322u, 0x000142BEu}}, \
     {7378u, 15387u, {0x4AF518C9u, 0x79C54F61u, 0x7F7279BAu, 0x00015AB3u}}, \
     {27462u, 9495u, {0xC98E25D0u, 0xC687FEF9u, 0xEA710C29u, 0x00018F8Fu}}, \
     {24125u, 22852u, {0xF069AEDEu, 0x4809A44Eu, 0x073981F1u, 0x0001B943u}}}
constexpr CrtGroup kCrtGroup[kCrtLevels][kCrtGroups] = {GPP_CRT_GROUPS};

// 1.5 2^23: a float of magnitude below 2^22 added to it is rounded to an
// integer in the low mantissa bits.
constexpr float kCrtMagic = 12582912.0f;

// The residues' constants of modulus p: 2^14, 2^28 and 2^42 mod p (symmetric),
// p and 1 / p.
struct CrtMod {
    float c1, c2, c3, p, inv;
};
__host__ __device__ constexpr int crt_sym_pow2(int k, int p) {
    int r = 1;
    for (int i = 0; i < k; ++i) r = r * 2 % p;
    return r > p / 2 ? r - p : r;
}
__host__ __device__ constexpr CrtMod crt_mod(int p) {
    return CrtMod{(float)crt_sym_pow2(14, p), (float)crt_sym_pow2(28, p),
                  (float)crt_sym_pow2(42, p), (float)p, 1.0f / (float)p};
}

// N = d0 + d1 2^14 + d2 2^28 + d3 2^42 with d0..d2 in [-8192, 8191] and
// |d3| <= 2^11 (2^15 for |N| up to 2^57: the sum of |d| times a residue's
// constants stays below 2^23), as floats built from their bits (no conversion
// instruction).
__host__ __device__ __forceinline__ void crt_digits(long long N, float (&d)[4]) {
    constexpr long long kBalance = 8192ll * (1 + (1ll << 14) + (1ll << 28));
    const long long M = N + kBalance;
    const int v[4] = {(int)(M & 16383) - 8192, (int)((M >> 14) & 16383) - 8192,
                      (int)((M >> 28) & 16383) - 8192, (int)(M >> 42)};
#pragma unroll
    for (int k = 0; k < 4; ++k) d[k] = small_int_to_float(v[k]);
}

// The same for |N| <= 2^bits, bits <= 41, in fewer digits: ND = 3 (the top one
// up to 2^13) or, for bits <= 18, ND = 2.
template <int ND>
__host__ __device__ __forceinline__ void crt_digits_n(long long N, float (&d)[ND]) {
    if constexpr (ND == 4) {
        crt_digits(N, d);
    } else if constexpr (ND == 3) {
        const long long M = N + 8192ll * (1 + (1ll << 14));
        d[0] = small_int_to_float((int)(M & 16383) - 8192);
        d[1] = small_int_to_float((int)((M >> 14) & 16383) - 8192);
        d[2] = small_int_to_float((int)(M >> 28));
    } else {
        const int M = (int)N + 8192;
        d[0] = small_int_to_float((M & 16383) - 8192);
        d[1] = small_int_to_float(M >> 14);
    }
}

// The digits of rint(scale (h + l)) of two normalised float-float values, for
// scale a power of two and scale |h + l| <= 2^53 (ND = 4), 2^41 (3) or 2^27 (2):
// each digit is rounded from the remainder and taken off its high part exactly
// (both are multiples of the smaller of the digit's weight and an ulp of h),
// so the last remainder is exact but for what lies below the integers.  A
// digit may pass its half range by two (2^41 + 2^29 below the top one).
template <int ND>
__host__ __device__ __forceinline__ void crt_digits_df2(const df2 &x, float scale, float2 (&d)[ND]) {
    const float2 magic = f2(kCrtMagic, kCrtMagic);
    float2 r = f2mul(x.h, f2(scale, scale));
    const float2 l = f2mul(x.l, f2(scale, scale));
#pragma unroll
    for (int k = ND - 1; k > 0; --k) {
        const float w = k == 3 ? 4398046511104.0f : k == 2 ? 268435456.0f : 16384.0f;  // 2^(14 k)
        const float2 v = k == ND - 1 ? r : f2add(r, l);
        d[k] = f2sub(f2fma(v, f2(1.0f / w, 1.0f / w), magic), magic);
        r = f2fma(d[k], f2(-w, -w), r);
    }
    d[0] = f2sub(f2add(f2add(r, l), magic), magic);
}

// v - p rint(v / p) on both lanes for integers |v| <= 2^23: the quotient is
// rounded once, from the product by a 1 / p whose relative error is at most
// 2^-25, so it is off by under 1 / (2 p) before rounding and the result is
// the symmetric residue, at most p / 2 in magnitude; all else is exact.
__host__ __device__ __forceinline__ float2 crt_reduce2(float2 v, float p, float inv) {
    const float2 magic = f2(kCrtMagic, kCrtMagic);
    const float2 q = f2sub(f2fma(v, f2(inv, inv), magic), magic);
    return f2fma(f2neg(q), f2(p, p), v);
}

// Symmetric residues mod m.p of two values with the digits d (lanes).
template <int ND>
__host__ __device__ __forceinline__ float2 crt_residue2(const float2 (&d)[ND], const CrtMod &m) {
    float2 v = d[0];
    if constexpr (ND > 1) v = f2fma(d[1], f2(m.c1, m.c1), v);
    if constexpr (ND > 2) v = f2fma(d[2], f2(m.c2, m.c2), v);
    if constexpr (ND > 3) v = f2fma(d[3], f2(m.c3, m.c3), v);
    return crt_reduce2(v, m.p, m.inv);
}

// The word-wise sum of t E over the groups, residues |r| <= 510 (each the
// true residue plus `bias`): t < 2^27, so the 64-bit words hold the sum of 8
// products.
struct CrtSum {
    unsigned long long a0 = 0, a1 = 0, a2 = 0;
    unsigned a3 = 0;
    template <int BIAS>
    __host__ __device__ __forceinline__ void add(int rp, int rq, const CrtGroup &g) {
        const unsigned t = (unsigned)rp * g.a + ((unsigned)rq * g.b + (512 - BIAS) * (g.a + g.b));
        a0 += (unsigned long long)t * g.E[0];
        a1 += (unsigned long long)t * g.E[1];
        a2 += (unsigned long long)t * g.E[2];
        a3 += t * g.E[3];
    }
};

// h 2^ex (h in [2^62, 2^64)) as a double, rounded to nearest.
__host__ __device__ __forceinline__ double crt_assemble(bool neg, unsigned long long h, int ex) {
    if (!(h >> 63)) {
        h <<= 1;
        --ex;
    }
    const unsigned long long m = (h >> 11) + ((h >> 10) & 1);  // up to 2^53
    const int E = ex + 63 + 1023;
    // The carry of a mantissa that rounds up to 2^53 moves the exponent field.
    if (E >= 1 && E <= 2045)
        return oz_double(((unsigned long long)neg << 63) +
                         (((unsigned long long)(E - 1) << 52) + m));
    const double r = (double)m * (neg ? -1.0 : 1.0);
#ifdef __CUDA_ARCH__
    return scalbn(r, E - 1075);
#else
    return __builtin_scalbn(r, E - 1075);
#endif
}

// |X| from the fraction's magnitude (w3..w0, most significant first) when its
// top word is zero.
#ifdef __CUDA_ARCH__
__device__ __noinline__
#else
inline
#endif
double crt_value_small(bool neg, unsigned w2, unsigned w1, unsigned w0, unsigned long long pn,
                       unsigned zero, int e) {
    unsigned long long hi = ((unsigned long long)w2 << 32) | w1, lo = (unsigned long long)w0 << 32;
    int n = 32;
    if (w2 == 0 && w1 == 0 && w0 < zero) return 0.0;
    while (!(hi >> 63)) {
        hi = (hi << 1) | (lo >> 63);
        lo <<= 1;
        ++n;
    }
#ifdef __CUDA_ARCH__
    const unsigned long long h = __umul64hi(hi, pn);
#else
    const unsigned long long h = (unsigned long long)(((unsigned __int128)hi * pn) >> 64);
#endif
    return crt_assemble(neg, h, e - n);
}

// X 2^e as a double, X the integer of magnitude below P / 2 with the given
// residues at level L: the sum is 2^128 X / P (mod 2^128) to within 2^26.5, at
// the wide level 2^26.7 (the rounding of the E), X to within 2^17 where the
// largest products are 2^106, 2^24.1 where they are 2^114 (a sum of that size
// is taken as 0); the top 64 bits of the fraction times P, rounded to nearest.
// Integer operations only, but for results outside the normal range.
template <int L>
__host__ __device__ __forceinline__ double crt_value(const CrtSum &s, int e) {
    constexpr unsigned long long pn = kCrtLevel[L].pn, off_hi = kCrtLevel[L].off_hi,
                                 off_lo = kCrtLevel[L].off_lo;
    e += kCrtLevel[L].pe;
    const unsigned long long l0 = s.a0 + off_lo;
    const unsigned long long c0 = l0 < s.a0 ? 1 : 0;
    const unsigned w0 = (unsigned)l0;
    unsigned long long l1 = (l0 >> 32) + (unsigned)s.a1;
    const unsigned w1 = (unsigned)l1;
    unsigned long long l2 = (l1 >> 32) + (s.a1 >> 32) + s.a2 + c0 + off_hi;
    const unsigned w2 = (unsigned)l2;
    // The upper words wrap as the 128-bit sum does.
    const unsigned w3 = (unsigned)(l2 >> 32) + s.a3;
    const bool neg = (int)w3 < 0;
    const unsigned x = neg ? 0xFFFFFFFFu : 0u;  // one's complement: off by one unit of 2^-128
    const unsigned v3 = w3 ^ x, v2 = w2 ^ x, v1 = w1 ^ x, v0 = w0 ^ x;
    if (v3 == 0) return crt_value_small(neg, v2, v1, v0, pn, kCrtLevel[L].zero, e);
#ifdef __CUDA_ARCH__
    const int z = __clz((int)v3);
    const unsigned long long hi =
        ((unsigned long long)__funnelshift_l(v2, v3, z) << 32) | __funnelshift_l(v1, v2, z);
    const unsigned long long h = __umul64hi(hi, pn);
#else
    const int z = __builtin_clz(v3);
    const unsigned long long up = ((unsigned long long)v3 << 32) | v2;
    const unsigned long long hi = z ? (up << z) | (v1 >> (32 - z)) : up;
    const unsigned long long h = (unsigned long long)(((unsigned __int128)hi * pn) >> 64);
#endif
    // |X| = hi 2^(64 - z) pn 2^pe / 2^128 = h 2^(pe - z)
    return crt_assemble(neg, h, e - z);
}

}  // namespace gpp
