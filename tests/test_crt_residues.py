"""The residue arithmetic of the tensor-core FP64 GEMM (gpp_crt.cuh), compiled
for the host from the header the kernels use: the moduli are pairwise coprime
and the products of each level's first moduli hold a 3M-form real or imaginary
part over 512 products of the level's integers; the float digits and residues of random and extreme integers
are exact and symmetric; the product sums' residues stay within the 2^23 that
the drain's reduction takes; and the value rebuilt from the residues of
re = P1 - P2 and im = P3 - P1 - P2 equals the exact 128-bit integer to its
rounding to a double (half a unit in the last place, plus the 2^17 that the
fraction's rounding, 2^26.1 of 2^128 / P = 2^10.2 units each way, and its
flush to zero may put it off, where the largest products are 2^106)."""
import os
import re
import shutil
import subprocess
from math import gcd

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "doe-csfg-hackathon_gb300", "csrc")

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include "gpp_crt.cuh"
using namespace gpp;

static unsigned long long st = 5;
static unsigned long long nx() {
    unsigned long long z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static long long draw(int kind, int bits) {
    const long long top = 1ll << bits;
    switch (kind) {
        case 0: return (long long)(nx() % (2 * (unsigned long long)top + 1)) - top;
        case 1: return nx() & 1 ? top : -top;
        case 2: return ((long long)(nx() % 2001) - 1000) % (top + 1);
        default: return (long long)(nx() % 3) - 1;
    }
}
template <int L>
static int check() {
    constexpr int NM = kCrtLevel[L].n;
    int bad = 0;
    for (int trial = 0; trial < 400; ++trial) {
        const int K = trial % 4 == 3 ? 512 : 1 + (int)(nx() % 512), kind = trial % 4;
        __int128 re = 0, im = 0;
        long long p[kCrtN][3] = {};
        for (int k = 0; k < K; ++k) {
            long long n[4];
            for (int t = 0; t < 4; ++t) n[t] = draw(trial < 8 ? 1 : kind == 1 && k % 3 ? 0 : kind, kCrtLevel[L].bits);
            re += (__int128)n[0] * n[2] - (__int128)n[1] * n[3];
            im += (__int128)n[0] * n[3] + (__int128)n[1] * n[2];
            float d[4][4];
            for (int t = 0; t < 4; ++t) {
                crt_digits(n[t], d[t]);
                if ((long long)d[t][0] + 16384ll * (long long)d[t][1] + (1ll << 28) * (long long)d[t][2] +
                        (1ll << 42) * (long long)d[t][3] != n[t]) ++bad;
            }
            for (int i = 0; i < NM; ++i) {
                const CrtMod m = crt_mod(kCrtModuli[i]);
                int r[6];
                for (int t = 0; t < 4; ++t) {
                    float2 dd[4];
                    for (int j = 0; j < 4; ++j) dd[j] = f2(d[t][j], -d[t][j]);
                    const float2 q = crt_residue2(dd, m);
                    r[t] = (int)q.x;
                    if (r[t] != q.x || 2 * abs(r[t]) > kCrtModuli[i] || (n[t] - r[t]) % kCrtModuli[i]) ++bad;
                    if ((-n[t] - (int)q.y) % kCrtModuli[i]) ++bad;
                }
                r[4] = (int)crt_reduce2(f2((float)(r[0] + r[1]), 0.f), m.p, m.inv).x;
                r[5] = (int)crt_reduce2(f2((float)(r[2] + r[3]), 0.f), m.p, m.inv).x;
                if (2 * abs(r[4]) > kCrtModuli[i] || 2 * abs(r[5]) > kCrtModuli[i]) ++bad;
                p[i][0] += r[0] * r[2];
                p[i][1] += r[1] * r[3];
                p[i][2] += r[4] * r[5];
            }
        }
        CrtSum sr, si;
        int rr[kCrtN + 1] = {}, ri[kCrtN + 1] = {};
        for (int i = 0; i < NM; ++i) {
            const CrtMod m = crt_mod(kCrtModuli[i]);
            int u[3];
            for (int g = 0; g < 3; ++g) {
                if (llabs(p[i][g]) > (1 << 23)) ++bad;
                u[g] = ((int)crt_reduce2(f2((float)p[i][g], 0.f), m.p, m.inv).x + 128) & 255;
            }
            rr[i] = u[0] - u[1];
            ri[i] = u[2] - u[0] - u[1];
        }
        for (int k = 0; k < (NM + 1) / 2; ++k) {
            sr.add<0>(rr[2 * k], rr[2 * k + 1], kCrtGroup[L][k]);
            si.add<-128>(ri[2 * k], ri[2 * k + 1], kCrtGroup[L][k]);
        }
        const CrtSum s[2] = {sr, si};
        const __int128 want[2] = {re, im};
        for (int t = 0; t < 2; ++t) {
            const double v = crt_value<L>(s[t], 0);
            const __int128 a = want[t] < 0 ? -want[t] : want[t];
            __int128 off = (__int128)v - want[t];
            if (off < 0) off = -off;
            if (off > (a >> 53) + (1 << 17)) {
                if (bad++ < 5) printf("trial %d: %a, off by %a\n", trial, v, (double)off);
            }
            // The scale: 2^e is exact, also into the subnormal range.
            if (crt_value<L>(s[t], -200) != std::ldexp(v, -200)) ++bad;
            if (crt_value<L>(s[t], -1100) != std::ldexp(v, -1100) && std::fabs(v) > 1e30) ++bad;
        }
    }
    return bad;
}
int main() {
    const int bad = check<0>() + check<1>() + check<2>() + check<3>();
    printf("%d failures\n", bad);
    return bad ? 1 : 0;
}
"""


def test_moduli_are_coprime_and_their_product_is_large_enough():
    text = open(os.path.join(CSRC, "gpp_crt.cuh")).read()
    m = re.search(r"#define GPP_CRT_MODULI \\\n([^\n]*)", text).group(1)
    p = [int(v) for v in m.split(",")]
    assert len(p) == 15 and max(p) <= 256
    assert all(gcd(a, b) == 1 for i, a in enumerate(p) for b in p[:i])
    for n, bits in re.findall(r"\{(\d+), (\d+), 0x[0-9A-F]{16}ull", text):
        product = 1
        for v in p[:int(n)]:
            product *= v
        assert 2 * 512 * 2 ** (2 * int(bits)) < product // 2


def test_residues_rebuild_exact_product_sums(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "crt_check.cu"
    src.write_text(HARNESS)
    exe = tmp_path / "crt_check"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-gencode",
                        "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "0 failures" in out.stdout
