"""The series' scratch (far_bytes of gpp_far.cu, called in the built library; no
GPU work) is bounded: at most 24 GB and, for the rows' weights and the list of
strays, one bands x ngpown complex array and half a byte a cell, for every size
that takes the series; states whose smallest pass would not fit do not take
it."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO
from gppsigma import build

CSRC = os.path.join(REPO, "doe-csfg-hackathon_gb300", "csrc")

SOURCE = r"""
#include <cstdio>
#include "gpp_far.h"
using namespace gpp;
int main() {
    const long long bands[] = {32, 130, 510, 2000, 4000, 20000, 80000, 340000};
    const long long rows[] = {16, 409, 1638, 6553, 60000};
    const long long cols[] = {512, 8192, 32768, 131072};
    const int freqs[] = {1, 3, 32, 2000, 30000};
    int bad = 0, taken = 0;
    for (int mixed = 0; mixed < 2; ++mixed)
        for (long long b : bands)
            for (long long r : rows)
                for (long long c : cols)
                    for (int w : freqs) {
                        Problem p{};
                        p.nb = (int)b;
                        p.ng = (int)r;
                        p.nc = (int)c;
                        p.nw = p.wx_stride = w;
                        if (!far_eligible(p, (int)b, mixed)) continue;
                        ++taken;
                        const double n = (double)far_bytes(p, (int)b, mixed);
                        const double most = 24.0 * (1ll << 30) + 16.0 * b * r + 0.5 * r * c;
                        if (n > most && bad++ < 10)
                            printf("%lld x %lld x %lld x %d mixed %d: %.1f GB\n", b, r, c, w, mixed, n / (1ll << 30));
                    }
    printf("%d sizes, %d over\n", taken, bad);
    return bad || taken < 100;
}
"""


def test_scratch_is_bounded(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    build.build()
    libdir = os.path.dirname(build.LIB)
    src = tmp_path / "bytes.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "bytes"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                        "-I", CSRC, "-I", os.path.join(REPO, "include"), str(src), "-o", str(exe),
                        "-L", libdir, "-lgpp_gb300", "-Xlinker", "-rpath," + libdir],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
