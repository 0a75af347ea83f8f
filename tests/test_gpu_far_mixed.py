"""The mixed-precision series of gpp_far.cu against the oracle, at the smallest
sizes that take it in that precision (the shapes of test_gpu_far_series.py take
it in FP64 only): ragged rows, columns and chunks, two to many frequencies a
band, strays, columns over decades, NaN and Inf.  That the device took the
series shows in its bits: they are not those of the per-term kernels, which the
same call runs when its scratch is refused (gpp_selftest_scratch_limit).

Norm-wise tolerance 1e-11: float-float terms are off by 2^-44 each and their sums
by about as much, with a hundred times that for sums that cancel."""
import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 1e-11
SHAPES = [  # nb, nv, ncouls, ngpown, nw, dw
    (64, 2, 20003, 40, 32, 0.25),
    (130, 3, 12289, 97, 8, 0.5),    # 127 bands: one short of a row tile
    (420, 0, 7937, 123, 3, 1.0),    # several row tiles
    (608, 8, 8001, 160, 2, 1.0),
]


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


def _inputs(shape, kind):
    nb, nv, nc, ng, nw, dw = shape
    inp = W.make_inputs(W.Shape(nb, nv, nc, ng, nw, dw=dw), 5 * nc + nw)
    rng = np.random.default_rng(nc)
    wt = inp.wtilde_array
    if kind == "strays":
        at = rng.uniform(size=wt.shape) < 0.004
        pick = inp.wx_array.ravel()[rng.integers(0, inp.wx_array.size, wt.shape)]
        off = rng.choice([1e-4, 0.3], wt.shape) * rng.uniform(-1, 1, wt.shape)
        wt[at] = (pick + off + 1e-5j)[at]
        wt[0, :3] = [300.0, 1.0 + 40.0j, -1e9]
    elif kind == "decades":
        fall = np.exp(-18.0 * np.arange(nc) / nc)
        inp.aqsntemp *= fall
        inp.I_eps_array *= fall
    return inp


def _run(d, n1):
    from gppsigma import ops
    lib = capi.load()
    lib.gpp_reset_launch_count()
    r = ops.sigma(d, "mixed", acht_n1=n1)
    ops.wait()
    return r, lib.gpp_launch_count()


@pytest.mark.parametrize("kind", ["band", "strays", "decades"])
@pytest.mark.parametrize("shape", SHAPES)
def test_mixed_series_against_the_oracle(shape, kind):
    import oracle_py
    from gppsigma import ops
    inp = _inputs(shape, kind)
    n1 = shape[4] >= 3
    d = ops.DeviceInputs.from_host(inp)
    r, launches = _run(d, n1)
    lib = capi.load()
    capi.check(lib.gpp_selftest_scratch_limit(512 << 20), "limit")
    try:
        t, few = _run(d, n1)
    finally:
        capi.check(lib.gpp_selftest_scratch_limit(0), "limit")
    assert launches > 20 > few
    # The series ran; with strays it pays at these sizes only where many
    # frequencies share its terms.
    if kind != "strays" or shape[4] == 32:
        assert not torch.equal(r.achtemp, t.achtemp)
    want = oracle_py.run(inp, "complex_seq", nthreads=8)
    for key in ["achtemp", "asxtemp"] + (["acht_n1_loc"] if n1 else []):
        w = want[key]
        for got in (r, t):
            g = getattr(got, key).cpu().numpy()
            assert np.max(np.abs(g - w)) <= TOL * max(np.max(np.abs(w)), 1e-300), key


def test_nan_and_inf_reach_what_they_reach_in_the_per_term_kernel():
    from gppsigma import ops
    inp = _inputs(SHAPES[0], "band")
    inp.wtilde_array[3, 100] = complex(np.nan, 0.0)
    r, launches = _run(ops.DeviceInputs.from_host(inp), True)
    assert launches > 20 and np.all(np.isnan(r.achtemp.cpu().numpy()))
    inp = _inputs(SHAPES[0], "band")
    inp.aqsntemp[40, 17] = complex(np.inf, 0.0)
    r, launches = _run(ops.DeviceInputs.from_host(inp), True)
    n1 = r.acht_n1_loc.cpu().numpy()
    assert launches > 20 and not np.isfinite(n1[40]) and np.isfinite(np.delete(n1, 40)).all()
    inp = _inputs(SHAPES[0], "band")
    inp.I_eps_array[7, 9] = complex(0.0, np.nan)
    r, launches = _run(ops.DeviceInputs.from_host(inp), True)
    assert launches > 20 and np.all(np.isnan(r.achtemp.cpu().numpy()))
