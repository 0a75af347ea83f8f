// gpp_crt_planes.cuh -- device code that forms residue planes of operands,
// shared by the kernels that read the operand (gpp_crt.cu) and that compute
// it (gpp_far.cu).
#pragma once

#include <cuda_bf16.h>

#include "gpp_crt.cuh"

namespace gpp {

constexpr int kExpZero = -4000;         // exponent of an all-zero chunk of a row
constexpr int kExpNonFinite = 1 << 20;  // of one that holds an Inf or a NaN

static __constant__ CrtMod c_crt_mod[kCrtN] = {
    crt_mod(256), crt_mod(255), crt_mod(253), crt_mod(251), crt_mod(247),
    crt_mod(241), crt_mod(239), crt_mod(233), crt_mod(229), crt_mod(227),
    crt_mod(223), crt_mod(217), crt_mod(211), crt_mod(199), crt_mod(197), crt_mod(193)};

// The e of frexp for the nonzero magnitude with bits b (b < 2^e).
__device__ __forceinline__ int crt_exponent(unsigned long long b) {
    if (b == 0) return kExpZero;
    const int E = (int)(b >> 52);
    if (E == 0x7FF) return kExpNonFinite;  // the bit patterns of Inf and NaN are the largest
    return E > 0 ? E - 1022 : (63 - __clzll((long long)b)) - 1073;
}

// Residues of 2 H consecutive k of a row, from the ND digits of re (dr) and
// im (di) in pairs of k, to the first nmod moduli: 4 H bytes per plane, at
// w + (g nmod + i) plane for g = re, im, re + im (H = 4: a core-matrix row).
template <int H, int ND>
__device__ __forceinline__ void crt_store_residues(const float2 (&dr)[H][ND], const float2 (&di)[H][ND],
                                                   int nmod, __nv_bfloat16 *w, size_t plane) {
#pragma unroll 1
    for (int i = 0; i < nmod; ++i) {
        const CrtMod m = c_crt_mod[i];
        unsigned v[3][H];
#pragma unroll
        for (int t = 0; t < H; ++t) {
            const float2 rr = crt_residue2(dr[t], m), ri = crt_residue2(di[t], m);
            const float2 rs = crt_reduce2(f2add(rr, ri), m.p, m.inv);
            const __nv_bfloat162 hr = __floats2bfloat162_rn(rr.x, rr.y);
            const __nv_bfloat162 hi = __floats2bfloat162_rn(ri.x, ri.y);
            const __nv_bfloat162 hs = __floats2bfloat162_rn(rs.x, rs.y);
            v[0][t] = *reinterpret_cast<const unsigned *>(&hr);
            v[1][t] = *reinterpret_cast<const unsigned *>(&hi);
            v[2][t] = *reinterpret_cast<const unsigned *>(&hs);
        }
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            __nv_bfloat16 *o = w + (size_t)(g * nmod + i) * plane;
            if constexpr (H == 4)
                *reinterpret_cast<uint4 *>(o) = make_uint4(v[g][0], v[g][1], v[g][2], v[g][3]);
            else
                *reinterpret_cast<uint2 *>(o) = make_uint2(v[g][0], v[g][1]);
        }
    }
}

}  // namespace gpp
