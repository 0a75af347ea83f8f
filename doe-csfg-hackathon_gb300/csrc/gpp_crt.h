// gpp_crt.h -- FP64-accurate complex GEMM on the tensor cores by residues
// (gpp_crt.cu); ozaki_zgemm chooses between it and the slicing of
// gpp_ozaki.cu.
#pragma once

#include "gpp_ozaki.h"

namespace gpp {

// As ozaki_bytes, ozaki_splits and ozaki_zgemm (gpp_ozaki.h).
size_t crt_bytes(int M, int N, int K, int splits);
int crt_splits(int K, int splits);
cudaError_t crt_zgemm(const OzOperand &X, const OzOperand &Y, int M, int N, int K, int splits,
                      double2 *Out, long long out_ld, long long split_stride, void *ws, int *err,
                      cudaStream_t s, cudaEvent_t after_slices);

// The passes of crt_zgemm on their own, for callers that keep or form operand
// planes themselves, at a level of precision (kCrtLevel); nothing is done
// where the device word `go`, if given, is 0.
//  crt_rows: residue planes sx [3 n][Mp][nc Kc] (bf16, core-matrix blocks) and
//    exponents ex [nc][Mp] of chunks [c0, c0 + nc) of X (Mp: rows, a multiple
//    of 128), row l being X's row order[l] if order is given; planes of Y are
//    the same in blocks of 256 rows.
//  crt_products: residues of the products of row tiles [mt0, mt0 + tiles) (128
//    rows each) with every row of Y: res [nc][3 n][Ms][Np] bytes.
//  crt_combine: Out[row0 + m][n] = (+=) the sum over the chunks.
// The last two stop at the first *rows (*live) rows of X, if given.
//  crt_sums: out [nc][Mp][Np], the products of single bf16 planes of each
//    operand (same blocks), summed in FP32 over each chunk.
constexpr int kCrtRowsX = 128, kCrtRowsY = 256, kCrtChunk = 512, kCrtBlockK = 64;
cudaError_t crt_rows(const OzOperand &X, const int *order, int Mp, int K, int Kc, int c0, int nc,
                     int level, void *sx, int *ex, const int *go, cudaStream_t s);
cudaError_t crt_products(const void *sx, const void *sy, int Mp, int Np, int Kc, int nc, int mt0,
                         int tiles, int level, unsigned char *res, int Ms, const int *go,
                         const int *rows, int *err, cudaStream_t s);
cudaError_t crt_sums(const void *sx, const void *sy, int Mp, int Np, int Kc, int nc, float *out,
                     const int *go, int *err, cudaStream_t s);
cudaError_t crt_combine(const unsigned char *res, const int *ex, const int *ey, int row0, int rows,
                        int Ms, int N, int Mp, int Np, int nc, int level, bool accumulate,
                        double2 *Out, long long out_ld, const int *go, const int *live,
                        cudaStream_t s);

}  // namespace gpp
