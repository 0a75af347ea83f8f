"""FP64 operands of the tensor-core GEMM keep 56 bits below the largest value of
a chunk, on the harness of test_gpu_ozaki.py: rows (1, then odd multiples of
2^-55 below 2^-34) against columns (0, 1, 1, ...) and the reverse, in both
layouts, give the sum of the small values exactly: 2^-31 to 2^-24 here, a
multiple of 2^-55 whose last place is 2^-84 or more, where the rebuilt value is
off by 2^-88 at most before it is rounded."""
import os
import shutil
import subprocess

import pytest

from gppsigma import build
from test_gpu_ozaki import CSRC, HARNESS, INCLUDE

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAIN = r"""
#include <cstdlib>
static int small_values(int M, int N, int K, bool kfast, bool swap) {
    std::vector<double2> big((size_t)(swap ? N : M) * K), one((size_t)(swap ? M : N) * K);
    const int nb = swap ? N : M, no = swap ? M : N;
    auto at = [&](std::vector<double2> &v, int l, int k, int L) -> double2 & {
        return v[kfast ? (size_t)l * K + k : (size_t)k * L + l];
    };
    for (int l = 0; l < nb; ++l)
        for (int k = 0; k < K; ++k)
            at(big, l, k, nb) = k == 0 ? make_double2(1.0, -1.0)
                                       : make_double2((2 * ((l * 7919 + k * 104729) % 1000003) + 1) * 0x1p-55,
                                                    -(2 * ((l * 611953 + k * 15485) % 1000003) + 1) * 0x1p-55);
    for (int l = 0; l < no; ++l)
        for (int k = 0; k < K; ++k) at(one, l, k, no) = make_double2(k == 0 ? 0.0 : 1.0, 0.0);
    const std::vector<double2> &x = swap ? one : big, &y = swap ? big : one;
    double2 *dx, *dy, *dout;
    int *err;
    void *ws;
    cudaMalloc(&dx, x.size() * 16); cudaMalloc(&dy, y.size() * 16);
    cudaMalloc(&dout, (size_t)M * N * 16); cudaMalloc(&err, 4); cudaMemset(err, 0, 4);
    cudaMalloc(&ws, gpp::ozaki_bytes(M, N, K, 1));
    cudaMemcpy(dx, x.data(), x.size() * 16, cudaMemcpyHostToDevice);
    cudaMemcpy(dy, y.data(), y.size() * 16, cudaMemcpyHostToDevice);
    const gpp::OzOperand X{dx, kfast ? K : M, kfast, M}, Y{dy, kfast ? K : N, kfast, N};
    if (gpp::ozaki_zgemm(X, Y, M, N, K, 1, dout, N, 0, ws, err, 0) != cudaSuccess) return 1;
    std::vector<double2> o((size_t)M * N);
    if (cudaMemcpy(o.data(), dout, o.size() * 16, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    int bad = 0;
    for (int m = 0; m < M; ++m)
        for (int n = 0; n < N; ++n) {
            double re = 0, im = 0;
            for (int k = 1; k < K; ++k) {
                const double2 v = at(big, swap ? n : m, k, nb);
                re += v.x;  // exact
                im += v.y;
            }
            if (o[(size_t)m * N + n].x != re || o[(size_t)m * N + n].y != im) ++bad;
        }
    printf("%d x %d x %d kfast %d swap %d: %d bad\n", M, N, K, kfast, swap, bad);
    cudaFree(dx); cudaFree(dy); cudaFree(dout); cudaFree(err); cudaFree(ws);
    return bad ? 1 : 0;
}
int main() {
    int bad = 0;
    for (int kfast = 0; kfast < 2; ++kfast)
        for (int swap = 0; swap < 2; ++swap) {
            bad |= small_values(3, 5, 40, kfast, swap);
            bad |= small_values(129, 257, 512, kfast, swap);
        }
    printf("%s\n", bad ? "FAILED" : "all ok");
    return bad;
}
"""


def test_small_values_beside_a_large_one_are_exact(tmp_path):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    libdir = os.path.dirname(build.LIB)
    src = tmp_path / "bits.cu"
    src.write_text(HARNESS[:HARNESS.index("int main()")] + MAIN)
    exe = tmp_path / "bits"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                        "-I", CSRC, "-I", INCLUDE, str(src), "-o", str(exe), "-L", libdir,
                        "-lgpp_gb300", "-Xlinker", "-rpath," + libdir],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "all ok" in out.stdout, out.stdout + out.stderr
