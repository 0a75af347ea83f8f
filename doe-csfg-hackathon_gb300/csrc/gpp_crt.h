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

}  // namespace gpp
