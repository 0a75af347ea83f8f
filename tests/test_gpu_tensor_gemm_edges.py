"""The residue GEMM (gpp_crt.cu) at the edges of its tiles, chunks and passes,
on the harness of test_gpu_ozaki.py: one row and column, one less and one more
than a row tile (128), a column tile (256) and a k chunk (512, and blocks of
64), several chunks in several splits, both layouts, and the same again in
passes of the smallest size (a 1 MB budget), which must keep the bits.  The
slices (GPP_TENSOR_GEMM=slices) run the same products as an independent check
within the same bound (1e-13 of the largest result)."""
import os
import shutil
import subprocess

import pytest

from gppsigma import build
from test_gpu_ozaki import CSRC, HARNESS, INCLUDE

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MAIN = r"""
int main() {
    int bad = 0;
    bad |= run(1, 1, 1, 1, false, 0, false);
    bad |= run(1, 257, 63, 1, true, 0, false);
    bad |= run(127, 255, 64, 1, false, 0, false);
    bad |= run(128, 256, 512, 1, true, 0, false);
    bad |= run(129, 513, 513, 1, false, 4, false);
    bad |= run(300, 70, 1025, 2, true, 8, false);
    bad |= run(257, 40, 1600, 1, false, 0, true);
    bad |= run(5, 900, 577, 3, true, 0, false);
    bad |= run_exact(129, 257, 513, false, 13);
    bad |= run_nonfinite();
    printf("%s\n", bad ? "FAILED" : "all ok");
    return bad;
}
"""


def test_tile_chunk_and_pass_edges(tmp_path):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    libdir = os.path.dirname(build.LIB)
    src = tmp_path / "edges.cu"
    src.write_text(HARNESS[:HARNESS.index("int main()")] + MAIN)
    exe = tmp_path / "edges"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                        "-I", CSRC, "-I", INCLUDE, str(src), "-o", str(exe), "-L", libdir,
                        "-lgpp_gb300", "-Xlinker", "-rpath," + libdir],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

    def go(**env):
        out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600,
                             env=dict(os.environ, **env))
        assert out.returncode == 0 and "all ok" in out.stdout, out.stdout + out.stderr
        return out.stdout

    assert go() == go(GPP_OZAKI_FOLD_MB="1")
    go(GPP_TENSOR_GEMM="slices")
