"""The digits of float-float values (crt_digits_df2 of gpp_crt.cuh), compiled
for the host: for random normalised h + l at every level's scale, signs and
binades from the largest value down to far below one, and values next to the
halves where a digit changes, the digits add up to an integer within one half
(and 2^-9, the rounding of the last remainder and of this check) of scale (h + l), and the
sum of digits times constants that a residue is reduced from stays below 2^23."""
import os
import shutil
import subprocess

import pytest

from test_crt_residues import CSRC

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "gpp_crt.cuh"
using namespace gpp;
static std::mt19937_64 rng(17);
static int bad = 0;
template <int ND> void one(float2 h, float2 l, float scale) {
    float2 d[ND];
    crt_digits_df2<ND>(df2{h, l}, scale, d);
    for (int lane = 0; lane < 2; ++lane) {
        const long double x = ((long double)(lane ? h.y : h.x) + (lane ? l.y : l.x)) * scale;
        long double n = 0, w = 1;
        float sum = 0;
        for (int k = 0; k < ND; ++k, w *= 16384) {
            const float v = lane ? d[k].y : d[k].x;
            if (v != std::rint(v)) ++bad;
            n += w * v;
            sum += std::fabs(v) * (k == 0 ? 1.f : 128.f);  // the residues' constants are at most 128
        }
        if (sum > 8388608.f) ++bad;
        long double off = n - x;
        if (off < 0) off = -off;
        if (off > (long double)(0.5 + 0.001953125)) {
            if (bad++ < 5) printf("ND %d: %.9g + %.9g scale %g off %g\n", ND, lane ? h.y : h.x, lane ? l.y : l.x, scale, (double)off);
        }
    }
}
// A normalised pair of magnitude below 1.
static void pair(float &h, float &l, int bits) {
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    double x = std::ldexp(u(rng), -(int)(rng() % (bits + 6)));
    if (rng() % 4 == 0) {  // next to k + 1/2 digits of some weight
        const int at = 14 * (1 + (int)(rng() % 3));
        const double s = std::ldexp(1.0, bits - at);
        x = (std::floor(x * s) + 0.5) / s + std::ldexp(u(rng), -(int)(rng() % 60) - 2);
        if (std::fabs(x) >= 1.0) x = 0.5;
    }
    h = (float)x;
    if (std::fabs(h) >= 1.0f) h = 0.75f;
    l = (float)(x - h);
    if (std::fabs(l) > std::ldexp(1.0f, std::ilogb(h) - 24)) l = 0.f;
}
template <int ND> void level(int bits) {
    for (int t = 0; t < 200000; ++t) {
        float2 h, l;
        pair(h.x, l.x, bits);
        pair(h.y, l.y, bits);
        one<ND>(h, l, std::ldexp(1.0f, bits));
    }
    const float one_ = 0x1.fffffep-1f;
    one<ND>(f2(one_, -one_), f2(0x1p-25f, -0x1p-25f), std::ldexp(1.0f, bits));
    one<ND>(f2(0.f, -0.f), f2(0.f, 0.f), std::ldexp(1.0f, bits));
}
int main() {
    level<4>(53);
    level<3>(41);
    level<3>(30);
    level<2>(18);
    printf("%d failures\n", bad);
    return bad ? 1 : 0;
}
"""


def test_digits_of_float_float_values(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "digits.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "digits"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-gencode",
                        "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
