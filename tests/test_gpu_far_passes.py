"""The series (gpp_far.cu) in the smallest passes: GPP_SERIES_PASS_MB=1 cuts a
state into groups of 8 rows, slabs of one chunk (an odd number of them, a ragged
last one), near passes of a few row pairs and planes of X per slab; the results
equal those of one pass to the rounding of the sums over groups (2^-49 of the
largest), and the per-term sums to the suites' tolerances."""
import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = [  # nb, nv, ncouls, ngpown, nw, dw, precision
    (64, 2, 5003, 17, 32, 0.25, "fp64"),     # 10 chunks; 3 groups of rows
    (300, 0, 2600, 41, 5, 0.5, "fp64"),      # 6 chunks, several row tiles
    (64, 2, 20003, 40, 32, 0.25, "mixed"),   # 40 chunks; 5 groups
    (700, 3, 4700, 150, 3, 1.0, "mixed"),    # 10 chunks, 19 groups
    (700, 0, 8000, 60, 1, 1.0, "fp64"),      # one frequency a band
]


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


@pytest.mark.parametrize("nb,nv,nc,ng,nw,dw,precision", CASES)
def test_smallest_passes_give_the_same_sums(monkeypatch, nb, nv, nc, ng, nw, dw, precision):
    import oracle_py
    from gppsigma import ops
    inp = W.make_inputs(W.Shape(nb, nv, nc, ng, nw, dw=dw), nc)
    inp.wtilde_array[::3, ::70] = 40.0 + 3.0j  # strays
    d = ops.DeviceInputs.from_host(inp)
    lib = capi.load()

    keys = ["achtemp", "asxtemp"] + (["acht_n1_loc"] if nw >= 3 else [])

    def go():
        lib.gpp_reset_launch_count()
        r = ops.sigma(d, precision, acht_n1=nw >= 3)
        ops.wait()
        return [getattr(r, k).cpu().numpy() for k in keys], lib.gpp_launch_count()

    capi.check(lib.gpp_selftest_scratch_limit(200 << 20), "limit")
    per_term, _ = go()
    capi.check(lib.gpp_selftest_scratch_limit(0), "limit")
    one, launches = go()
    monkeypatch.setenv("GPP_SERIES_PASS_MB", "1")
    many, more = go()
    again, _ = go()
    monkeypatch.delenv("GPP_SERIES_PASS_MB")
    assert launches > 20 and more > 5 * launches
    assert not np.array_equal(one[0], per_term[0])  # the series ran
    want = oracle_py.run(inp, "complex_seq", nthreads=8)
    tol = 1e-12 if precision == "fp64" else 1e-8
    for a, b, c, k in zip(one, many, again, keys):
        assert np.array_equal(b, c)
        assert np.max(np.abs(a - b)) <= 2.0 ** -49 * np.max(np.abs(a)) * (16 if k == "achtemp" else 1), k
        assert np.max(np.abs(b - want[k])) <= tol * np.max(np.abs(want[k])), k
