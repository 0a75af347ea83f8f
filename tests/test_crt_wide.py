"""The wide level of the residue arithmetic (gpp_crt.cuh), which stands for the
FP64 operands of the tensor-core GEMM: its integers hold at least the 56 bits
that the slices of gpp_ozaki_split.cuh hold, its 16 moduli are pairwise coprime
and their product holds the sums; digits, residues and the value rebuilt from
them are those of exact 128-bit arithmetic (the harness of
test_crt_residues.py at the wide level), to half a unit in the last place plus
2^25: the rounding of the fractions, 2^26.7 of 2^128 / P = 2^2.6 units each way
(2^24.1), and the flush to zero of such a sum."""
import os
import re
import shutil
import subprocess
from math import gcd

import pytest

from test_crt_residues import CSRC, HARNESS


def test_the_wide_level_holds_what_the_slices_hold():
    text = open(os.path.join(CSRC, "gpp_crt.cuh")).read()
    p = [int(v) for v in re.search(r"#define GPP_CRT_MODULI \\\n([^\n]*)", text).group(1).split(",")]
    p.append(int(re.search(r"kCrtModuli\[kCrtN\] = \{GPP_CRT_MODULI, (\d+)\}", text).group(1)))
    assert len(p) == 16 == int(re.search(r"kCrtN = (\d+);", text).group(1))
    assert all(gcd(a, b) == 1 for i, a in enumerate(p) for b in p[:i])
    bits = int(re.search(r"kCrtWideBits = (\d+);", text).group(1))
    slices = int(re.search(r"kOzSlices = (\d+);",
                           open(os.path.join(CSRC, "gpp_ozaki_split.cuh")).read()).group(1))
    product = 1
    for v in p:
        product *= v
    assert bits >= 7 * slices and 2 * 512 * 2 ** (2 * bits) < product // 2
    gemm = open(os.path.join(CSRC, "gpp_crt.cu")).read()
    zgemm = gemm[gemm.index("cudaError_t crt_zgemm"):]
    assert zgemm.count("kCrtWide") == 3  # operand planes, products and combination


def test_the_wide_level_rebuilds_exact_product_sums(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    main = HARNESS.index("int main()")
    source = (HARNESS[:main].replace("(1 << 17)", "(1 << 25)") + """
int main() {
    const int bad = check<kCrtWide>();
    printf("%d failures\\n", bad);
    return bad ? 1 : 0;
}
""")
    src = tmp_path / "crt_wide.cu"
    src.write_text(source)
    exe = tmp_path / "crt_wide"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-gencode",
                        "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "0 failures" in out.stdout, out.stdout + out.stderr
